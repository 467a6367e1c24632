"""What a candidate sweep reports of itself, with the simulations left out: the bytes
of the kernel its candidates take, and no time spent on choosing what does not act on
them."""
from __future__ import annotations

import importlib
import types

import numpy as np
import pytest


class FakeGrid:
    t, nx, ny, nz = None, 256, 128, 96

    def close(self):
        pass


class FakeSlot:
    def __init__(self, fd):
        self.grid = FakeGrid()

    def prepare(self, cand, variant=0, retire=None):
        self.cand, self.shape, self.dt = cand, (256, 128, cand["nz"]), 1.0

    def start(self):
        pass

    def amplitudes(self):
        return np.ones(11, complex)

    def close(self):
        pass


@pytest.fixture
def B(monkeypatch):
    batch = importlib.import_module("3d_fdtd_b200.batch")
    monkeypatch.setattr(batch, "Slot", FakeSlot)
    monkeypatch.setattr(batch, "_sweep_call", lambda *a: None)
    return batch


@pytest.fixture
def engine(fd):
    return types.SimpleNamespace(lib=types.SimpleNamespace(timefield3d_zero_fields=lambda t: None), YEE_AUTO=0,
                                 YEE_FLAT=fd.YEE_FLAT, YEE_FLAT4=fd.YEE_FLAT4, YEE_FUSED=fd.YEE_FUSED,
                                 YEE_WAVE=fd.YEE_WAVE, YEE_STREAM=fd.YEE_STREAM)


def moved(cands, cell):
    """48 B of fields and the coefficients a cell, 32 B a cell and slab."""
    return sum((cell * 256 * 128 * c["nz"] + 32 * 24 * (128 * c["nz"] + 256 * c["nz"] + 256 * 128)) * c["steps"]
               for c in cands)


def test_sweep_bytes_are_the_kernels(engine, B):
    cands = B.candidates(3, seed=2)
    assert B.sweep_persistent(engine, cands, group=2, shape=(0, 2.0))["bytes"] == moved(cands, 52)
    assert B.sweep(engine, cands, slots=2, variant=engine.YEE_STREAM)["bytes"] == moved(cands, 52)
    assert B.sweep(engine, cands, slots=2, variant=engine.YEE_FLAT4)["bytes"] == moved(cands, 60)


def test_sweep_times_no_tile_shapes(engine, B, monkeypatch):
    # candidates come from the rasterisers: fdtd_sweep_run gives them streams of their own,
    # which its tile shape does not touch
    def tune(*a, **k):
        raise AssertionError("tile shapes timed")

    monkeypatch.setattr(B, "autotune_tiles", tune)
    r = B.sweep_persistent(engine, B.candidates(2, seed=2), group=2)
    assert sorted(r["results"]) == [0, 1] and r["tuning"] == {}
