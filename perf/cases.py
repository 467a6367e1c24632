"""The work users of this package have it do, as measurable cases.

Each case is a dict of plain values; `kind` says which public calls it makes:

  run      a forward simulation in one timefield3d_run: Si strip taper (spline widths, sub-pixel fill), CPML, scheduled
           mode pulse, two overlap monitors.  FP32 for design work, FP64 for validating it; optionally a lossy core.
  dipole   plain stepwise FDTD: a soft point source driven from the host before every timefield3d_apply_timestep_omp_full,
           Mur boundary, FP64, probes recorded on the device.
  driver   one design iteration written like the reference's own program: per step a mode source, a step, a y-slice DFT,
           three mode overlaps read back, an edge store; then the adjoint run and the permittivity gradient.  FP64, Mur.
  adjoint  the exact gradient of the transmission with respect to a taper's control widths: forward run, adjoint run, both
           with their edge fields stored, and the reduction.  FP32.
  sweep    several candidate tapers of uneven length advanced together by fdtd_sweep_run.  FP32.
  mode     the fundamental mode of a strip cross-section (FP64 Arnoldi solver), as every design run needs for its source.
  train    fine-tuning the surrogate network on the designs simulated so far (one epoch of minibatches).
  query    one ascent step of the surrogate's proposals: predicted spectra of a set of designs, and their input gradient.

Fields of FP32 runs are returned as FP32 (the host mirror widens them to doubles), and so are sums formed from them.
"""
import ctypes as C
import importlib
import math

import numpy as np
import torch

fd = importlib.import_module("3d_fdtd_b200")

DP, FP = C.POINTER(C.c_double), C.POINTER(C.c_float)
PI = fd.REF_PI
EP_CLAD, EP_CORE = 2.085, 12.1
LAM0, BANDWIDTH = 1.55, 0.3
NCTRL = 20


def listed():
    return [
        # the benchmark's Si taper: one design simulation, the package's main use
        dict(name="taper_f32", kind="run", nx=200, ny=160, nz=400, cells=12, precision="f32", steps=1024, waves=11,
             lossy=False, fields=False),
        # the same grid on the FP64 path that FP32 results are validated against
        dict(name="taper_f64", kind="run", nx=200, ny=160, nz=400, cells=12, precision="f64", steps=128, waves=11,
             lossy=False, fields=False),
        # a wide device window: long rows, the largest grid
        dict(name="wide_f32", kind="run", nx=384, ny=256, nz=384, cells=12, precision="f32", steps=192, waves=11,
             lossy=False, fields=False),
        # a window cut to a device's own size, no dimension a multiple of four
        dict(name="ragged_f32", kind="run", nx=157, ny=131, nz=203, cells=10, precision="f32", steps=512, waves=5,
             lossy=False, fields=False),
        # a small exploratory run with conductivity, all fields looked at afterwards
        dict(name="small_lossy_f32", kind="run", nx=96, ny=80, nz=64, cells=8, precision="f32", steps=256, waves=3,
             lossy=True, fields=True),
        # the 64^3 dipole of the tests: stepwise calls, launch-bound
        dict(name="dipole_f64", kind="dipole", n=64, steps=400),
        # a drop-in program's design iteration on the tests' small taper
        dict(name="driver_f64", kind="driver", nx=40, ny=28, nz=72, steps=100),
        # the optimiser's exact gradient on a member of the candidate family
        dict(name="adjoint_f32", kind="adjoint", nx=256, ny=128, nz=128, cells=12, steps=1024),
        # eight candidates of the 64-candidate family, lengths 5 to 20 um
        dict(name="sweep_f32", kind="sweep", nx=256, ny=128, count=8, steps=160),
        # the TE0 mode of the candidates' input strip
        dict(name="mode_f64", kind="mode", mi=200, mj=160, krylov=20, tol=1e-8),
        # the optimiser's fine-tuning and proposal steps
        dict(name="train", kind="train", designs=1024, batch=128),
        dict(name="query", kind="query", rows=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "dipole", "driver", "adjoint", "sweep", "mode", "train", "query"])
    if kind == "run":
        f64 = rng.random() < 0.3
        L = rng.choice([6, 8, 10, 12, 16])
        nx, ny, nz = (_log_int(rng, lo, hi) for lo, hi in ((64, 400), (56, 256), (72, 400)))
        if rng.random() < 0.5:
            nx -= nx % 4
        cells = nx * ny * nz
        steps = max(32, min(1024, int((2.0e9 if f64 else 5.0e9) / cells)))
        fields = cells < 1_000_000
        if fields:   # looked at while the pulse is inside the window
            steps = min(steps, 256)
        return dict(kind="run", nx=nx, ny=ny, nz=nz, cells=L, precision="f64" if f64 else "f32", steps=steps,
                    waves=rng.choice([1, 3, 5, 11]), lossy=rng.random() < 0.25, fields=fields)
    if kind == "dipole":
        n = _log_int(rng, 24, 96)
        return dict(kind="dipole", n=n, steps=_log_int(rng, 50, 400))
    if kind == "driver":
        return dict(kind="driver", nx=rng.randint(32, 64), ny=rng.randint(24, 48), nz=rng.randint(60, 110),
                    steps=_log_int(rng, 30, 100))
    if kind == "adjoint":
        return dict(kind="adjoint", nx=4 * rng.randint(24, 64), ny=rng.randint(64, 128), nz=rng.randint(96, 128),
                    cells=rng.choice([8, 10, 12]), steps=rng.randint(640, 1024))   # the pulse has to reach the end
    if kind == "sweep":
        return dict(kind="sweep", nx=4 * rng.randint(32, 64), ny=rng.randint(72, 128), count=rng.randint(2, 8),
                    steps=_log_int(rng, 40, 160))
    if kind == "mode":
        return dict(kind="mode", mi=_log_int(rng, 64, 256), mj=_log_int(rng, 48, 160), krylov=20, tol=1e-8)
    if kind == "train":
        batch = 8 * rng.randint(4, 32)
        return dict(kind="train", designs=batch * rng.randint(2, 8) + rng.randint(0, 40), batch=batch)
    return dict(kind="query", rows=_log_int(rng, 4, 512))


# ---------------------------------------------------------------------------
# inputs, from the seed alone (numpy only: prepare and exact share them)
# ---------------------------------------------------------------------------
def _dims(case):
    if case["kind"] == "dipole":
        return case["n"], case["n"], case["n"]
    return case["nx"], case["ny"], case["nz"]


def _profile(nx, ny, half_w, half_h, cy, seed):
    """A quasi-TE guided profile on the whole cross-section, [ny][nx][6] complex (as a mode file holds it)."""
    rng = np.random.default_rng(seed)
    x = np.arange(nx)[None, :] - nx // 2 + rng.uniform(-0.4, 0.4)
    y = np.arange(ny)[:, None] - cy + rng.uniform(-0.4, 0.4)
    wx, wy = 0.9 * half_w * rng.uniform(0.9, 1.1), 1.1 * half_h * rng.uniform(0.9, 1.1)
    g = np.exp(-np.abs(x / wx) ** 1.7 - np.abs(y / wy) ** 1.5)
    n = rng.uniform(2.3, 2.8)
    f = np.zeros((ny, nx, 6), complex)
    f[..., 0] = g * (1 + 0.02j * x / nx)
    f[..., 1] = 0.03 * g * (x / wx) * (y / wy)
    f[..., 2] = 0.3j * g * x / wx
    f[..., 3] = -n * f[..., 1] + 0.01j * g
    f[..., 4] = n * f[..., 0]
    f[..., 5] = 0.25j * g * y / wy
    return f


def _pulse(steps, dt):
    w0 = 2 * PI / LAM0
    dw = 2 * math.pi * BANDWIDTH / LAM0 ** 2
    sigma = min((2 * math.sqrt(2 * math.log(2)) / dw) / dt, steps / 10)   # short runs: a shorter pulse
    n = np.arange(steps, dtype=np.float64)
    return np.exp(-((n - 3 * sigma) ** 2) / (2 * sigma ** 2)), n * dt * w0


def _taper(case, seed):
    """Geometry, modes and source of the taper kinds (one candidate)."""
    nx, ny, nz = _dims(case)
    L, dx = case["cells"], 0.025
    rng = np.random.default_rng(seed)
    cx, cy = nx // 2, ny // 2
    half = max(2, min(4, ny // 16))
    w_in, w_out = 2 * max(4, nx // 20), 2 * int(0.3 * nx)
    z0, z1 = L + 18, nz - L - 18
    widths = np.sort(rng.uniform(w_in * dx, w_out * dx, NCTRL))
    dt = 0.99 * dx / math.sqrt(3)
    amp, phase = _pulse(case["steps"], dt)
    waves = case.get("waves", 11)
    lams = [1.55] if waves == 1 else [1.50 + 0.1 * i / (waves - 1) for i in range(waves)]
    return dict(nx=nx, ny=ny, nz=nz, L=L, dx=dx, dt=dt, cx=cx, cy=cy, rows=(cy - half, cy + half + 1),
                w_in=(cx - w_in // 2, cx + w_in // 2), w_out=(cx - w_out // 2, cx + w_out // 2), z0=z0, z1=z1,
                widths=widths, amp=amp, phase=phase, omega=np.array([2 * PI / l for l in lams]),
                src_z=L + 8, launch_z=L + 13, out_z=nz - L - 8, steps=case["steps"],
                mode_in=_profile(nx, ny, w_in / 2, half + 0.5, cy, 2 * seed + 1),
                mode_out=_profile(nx, ny, w_out / 2, half + 0.5, cy, 2 * seed + 2),
                sig=float(rng.uniform(0.05, 0.2)) if case.get("lossy") else 0.0,
                sig_box=(nx // 4, 3 * nx // 4, cy - half, cy + half + 1, nz // 3, 2 * nz // 3))


def _dipole(case, seed):
    n, dx = case["n"], 0.020
    rng = np.random.default_rng(seed)
    dt = 0.99 * dx / math.sqrt(3)
    amp, phase = _pulse(case["steps"], dt)
    a = n // 2 - n // 6
    pts = [tuple(int(v) for v in rng.integers(n // 8, n - n // 8, 3)) for _ in range(4)]
    src = tuple(int(n // 2 + v) for v in rng.integers(-2, 3, 3))
    return dict(nx=n, ny=n, nz=n, dx=dx, dt=dt, drive=amp * np.sin(phase), eps=float(np.float32(rng.uniform(2, 12))),
                cube=(a, a + n // 3), pts=pts, src=src)


def _driver(case, seed):
    nx, ny, nz = _dims(case)
    dx, T = 0.05, case["steps"]
    dt = 0.99 * dx / math.sqrt(3)
    rng = np.random.default_rng(seed)
    cx, cy, z0, z1 = nx // 2, ny // 2, nz // 3, 2 * nz // 3
    seg = 4
    left = [int(cx - v) for v in rng.integers(4, 8, seg + 1)]
    right = [int(cx + v) for v in rng.integers(4, 8, seg + 1)]
    n = np.arange(T)
    return dict(nx=nx, ny=ny, nz=nz, dx=dx, dt=dt, T=T, cx=cx, cy=cy, rows=(cy - 2, cy + 3), z0=z0, z1=z1, seg=seg,
                left=left, right=right, omega=2 * PI / LAM0, amp=np.exp(-((n - 0.3 * T) ** 2) / (2 * (0.1 * T) ** 2)),
                wg_in=(left[0], right[0]), wg_out=(left[-1], right[-1]), src_z=nz // 6, launch_z=nz // 6 + 4,
                out_z=nz - nz // 5, mode=_profile(nx, ny, 5, 2.5, cy, 2 * seed + 1))


def _sweep_cases(case, seed):
    """Candidates of uneven length: nz in [96, 384], step counts in proportion."""
    rng = np.random.default_rng(seed)
    nzs = np.linspace(100, 380, case["count"]).astype(int)   # the work does not depend on the seed
    rng.shuffle(nzs)
    return [dict(kind="run", nx=case["nx"], ny=case["ny"], nz=int(nz), cells=12, waves=11,
                 steps=int(case["steps"] * (0.5 + 0.5 * nz / 380))) for nz in nzs]


def _strip(case, seed):
    mi, mj = case["mi"], case["mj"]
    rng = np.random.default_rng(seed)
    w, h = int(rng.integers(18, 24)), 9
    return (mi // 2 - w // 2, mi // 2 - w // 2 + w, mj // 2 - h // 2, mj // 2 - h // 2 + h)


def _designs(n, seed):
    """Normalised widths and a smooth spectrum standing in for the simulated one: [n][20], [n][22]."""
    rng = np.random.default_rng(seed)
    x = ((np.sort(rng.uniform(0.5, 3.0, (n, NCTRL)), axis=1) - 1.75) / 1.25).astype(np.float32)
    a, b = rng.normal(size=(2, NCTRL, 22)) / math.sqrt(NCTRL)
    return x, (0.6 * np.sin(x @ a) + 0.3 * np.cos(x @ b)).astype(np.float32)


def _weights(seed):
    """Network parameters as a trained network has them: flat W1, b1, ..., W4, b4."""
    rng = np.random.default_rng(seed)
    out = []
    for o, i in ((256, NCTRL), (256, 256), (256, 256), (22, 256)):
        out += [rng.uniform(-1, 1, o * i) / math.sqrt(i), rng.uniform(-1, 1, o) / math.sqrt(i)]
    return np.concatenate(out).astype(np.float32)


# ---------------------------------------------------------------------------
# what a program keeps before the call
# ---------------------------------------------------------------------------
def _dptr(a):
    return a.ctypes.data_as(DP)


def _taper_grid(p, precision):
    g = fd.Grid(p["nx"], p["ny"], p["nz"], p["dx"], precision)
    t, (b, top) = g.t, p["rows"]
    fd.lib.timefield3d_set_background(t, EP_CLAD, 1.0)
    fd.lib.timefield3d_set_waveguide(t, EP_CORE, p["w_in"][0], p["w_in"][1], 0, p["z0"], b, top)
    fd.lib.timefield3d_set_waveguide(t, EP_CORE, p["w_out"][0], p["w_out"][1], p["z1"], p["nz"], b, top)
    fd.call("timefield3d_set_spline_taper", t, EP_CORE, 1.0, NCTRL, _dptr(p["widths"]), float(p["cx"]), p["z0"],
            p["z1"], b, top)
    if p["sig"]:
        fd.lib.timefield3d_set_prism_electric_conductivity(t, p["sig"], *p["sig_box"])
    fd.call("timefield3d_set_cpml", t, p["L"], 3, -1.0, 1.0, 0.0)
    return g


def _monitor(g, p, z, mode):
    return fd.call("timefield3d_add_overlap_monitor", g.t, p["cx"], p["cy"], z, mode.struct, 0, len(p["omega"]),
                   _dptr(p["omega"]))


def _schedule(g, p, mode):
    fd.call("timefield3d_set_source_schedule", g.t, p["cx"], p["cy"], p["src_z"], mode.struct, 0, 0, p["steps"],
            _dptr(p["amp"]), _dptr(p["phase"]))


def _simulation(p, precision):
    """A grid with its monitors and source schedule set up, materials on the device."""
    g = _taper_grid(p, precision)
    mons = [_monitor(g, p, p["launch_z"], fd.HostMode(p["mode_in"], p["dx"])),
            _monitor(g, p, p["out_z"], fd.HostMode(p["mode_out"], p["dx"]))]
    _schedule(g, p, fd.HostMode(p["mode_in"], p["dx"]))
    fd.call("timefield3d_upload_materials", g.t)
    return g, mons


def _read(g, mon, n):
    acc = np.zeros(n, np.complex128)
    fd.call("timefield3d_read_overlap_monitor", g.t, mon, acc.ctypes.data_as(C.POINTER(fd.Complex)))
    return acc


class State:
    """What a program holds between calls; frees the library's objects it made."""

    def __init__(self, case):
        self.case, self.free = case, []

    def __del__(self):
        for f in self.free:
            f()


def prepare(case, seed):
    s = State(case)
    kind = case["kind"]
    if kind == "run":
        s.p = _taper(case, seed)
        s.f32 = case["precision"] == "f32"
        s.g, s.mons = _simulation(s.p, fd.F32 if s.f32 else fd.F64)
        s.free.append(s.g.close)
    elif kind == "dipole":
        s.p = p = _dipole(case, seed)
        s.g = fd.Grid(p["nx"], p["ny"], p["nz"], p["dx"], fd.F64)
        s.free.append(s.g.close)
        a, b = p["cube"]
        fd.lib.timefield3d_set_background(s.g.t, 1.0, 1.0)
        fd.lib.timefield3d_set_prism_permittivity(s.g.t, p["eps"], a, b, a, b, a, b)
        s.probes = [fd.call("timefield3d_add_probe", s.g.t, *pt, m, case["steps"]) for pt in p["pts"] for m in range(3)]
        fd.call("timefield3d_upload_materials", s.g.t)
    elif kind == "driver":
        s.p = p = _driver(case, seed)
        s.g = g = fd.Grid(p["nx"], p["ny"], p["nz"], p["dx"], fd.F64)
        b, top = p["rows"]
        fd.lib.timefield3d_set_background(g.t, EP_CLAD, 1.0)
        fd.lib.timefield3d_set_waveguide(g.t, EP_CORE, p["wg_in"][0], p["wg_in"][1], 0, p["z0"], b, top)
        fd.lib.timefield3d_set_waveguide(g.t, EP_CORE, p["wg_out"][0], p["wg_out"][1], p["z1"], p["nz"], b, top)
        n = p["seg"] + 1
        s.taper = fd.call("adjoint3d_taper_new", EP_CORE, 1.0, p["seg"], p["z0"], p["z1"], (C.c_int * n)(*p["left"]),
                          (C.c_int * n)(*p["right"]), b, top, p["T"])
        fd.lib.adjoint3d_taper_insert(g.t, s.taper)
        s.launch, s.out = fd.HostMode(p["mode"], p["dx"]), fd.HostMode(p["mode"], p["dx"])
        for m in (s.launch, s.out):
            s.free.append(lambda m=m: fd.lib.timefield3d_release_mode(m.struct))
        s.free += [lambda: fd.lib.adjoint3d_taper_free(s_taper), g.close]
        s_taper = s.taper
    elif kind == "adjoint":
        s.p = p = _taper(case, seed)
        s.grids = []
        for _ in range(2):   # the forward and the adjoint simulation
            g = _taper_grid(p, fd.F32)
            fd.call("timefield3d_upload_materials", g.t)
            s.grids.append(g)
        s.omega = np.array([2 * PI / LAM0])
        _schedule(s.grids[0], p, fd.HostMode(p["mode_in"], p["dx"]))
        s.mode = fd.HostMode(p["mode_out"], p["dx"])
        s.mon = fd.call("timefield3d_add_overlap_monitor", s.grids[0].t, p["cx"], p["cy"], p["out_z"], s.mode.struct, 0,
                        1, _dptr(s.omega))
        s.store = fd.call("fdtd_spline_store_new", s.grids[0].t, NCTRL, _dptr(p["widths"]), float(p["cx"]), p["z0"],
                          p["z1"], p["rows"][0], p["rows"][1], p["steps"])
        store, grids = s.store, s.grids
        s.free += [lambda: fd.lib.fdtd_spline_store_free(store)] + [g.close for g in grids]
    elif kind == "sweep":
        s.ps = [_taper(c, 100 * seed + i) for i, c in enumerate(_sweep_cases(case, seed))]
        s.sims = [_simulation(p, fd.F32) for p in s.ps]
        s.free += [g.close for g, _ in s.sims]
    elif kind == "mode":
        s.core, s.seed = _strip(case, seed), seed
        s.modes = importlib.import_module("3d_fdtd_b200.modes")
        s.libc = C.CDLL(None)
    else:
        s.opt = importlib.import_module("3d_fdtd_b200.surrogate_opt")
        s.net = s.opt.Net(fd)
        s.free.append(s.net.close)
        s.w = _weights(seed)
        s.net.set_params(s.w)
        s.x, s.y = _designs(case["designs"] if kind == "train" else case["rows"], seed + 1)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    return _RUN[s.case["kind"]](s)


def _run_run(s):
    fd.lib.timefield3d_zero_fields(s.g.t)
    fd.call("timefield3d_run", s.g.t, s.p["dt"], s.p["steps"])
    acc = np.stack([_read(s.g, m, len(s.p["omega"])) for m in s.mons])
    out = {"monitors": acc.astype(np.complex64) if s.f32 else acc}
    if s.case["fields"]:
        f = s.g.fields()
        out["fields"] = f.astype(np.float32) if s.f32 else f
    return out


def _run_dipole(s):
    p, t = s.p, s.g.t
    fd.lib.timefield3d_zero_fields(t)
    i, j, k = p["src"]
    for v in p["drive"].tolist():
        fd.lib.timefield3d_set_source_value(t, i, j, k, 2, v)
        fd.lib.timefield3d_apply_timestep_omp_full(t, p["dt"])
    fd.check("steps")
    out = np.zeros((len(s.probes), len(p["drive"])))
    for q, pid in enumerate(s.probes):
        fd.call("timefield3d_read_probe", t, pid, _dptr(out[q]), out.shape[1])
    return out


def _run_driver(s):
    p, t, lib, dt = s.p, s.g.t, fd.lib, s.p["dt"]
    cx, cy, T = p["cx"], p["cy"], p["T"]
    lib.timefield3d_zero_fields(t)
    cum = [fd.Complex() for _ in range(3)]
    for n in range(T):
        phase = n * dt * p["omega"]
        lib.timefield3d_mode_source(t, cx, cy, p["src_z"], s.launch.struct, phase, p["amp"][n], 0)
        lib.timefield3d_apply_timestep_omp_full(t, dt)
        lib.timefield3d_update_fourier_fields_y_slice_omp(t, phase, cy)
        lib.timefield3d_mode_overlap(t, cx, cy, p["launch_z"], s.launch.struct, phase, 0, C.byref(cum[0]))
        lib.timefield3d_mode_overlap(t, cx, cy, p["launch_z"], s.launch.struct, phase, 1, C.byref(cum[1]))
        lib.timefield3d_mode_overlap(t, cx, cy, p["out_z"], s.out.struct, phase, 0, C.byref(cum[2]))
        lib.adjoint3d_taper_store_forward_fields(s.taper, t, n)
    fd.check("forward")
    fields = s.g.fields()
    fourier = s.g.fourier()[:, cy]
    lib.timefield3d_zero_fields(t)
    for n in range(T - 1, -1, -1):
        lib.timefield3d_mode_source_adjoint(t, cx, cy, p["out_z"], s.out.struct, (n + 1) * dt * p["omega"], 0)
        lib.timefield3d_apply_timestep_omp_full(t, dt)
        lib.adjoint3d_taper_store_adjoint_fields(s.taper, t, n)
    lib.adjoint3d_taper_calculate_ep_gradient(s.taper)
    lib.adjoint3d_taper_calculate_gradients_from_ep_gradient(s.taper, EP_CORE - EP_CLAD)
    fd.check("adjoint")
    cells = 2 * (p["rows"][1] - p["rows"][0]) * (p["z1"] - p["z0"])
    return {"overlaps": np.array([complex(c.re, c.im) for c in cum]), "fields": fields, "fourier": fourier.copy(),
            "gradient": np.ctypeslib.as_array(s.taper.ep_gradient, shape=(cells,)).copy()}


def _run_adjoint(s):
    p, (gf, ga) = s.p, s.grids
    fd.lib.timefield3d_zero_fields(gf.t)
    fd.call("fdtd_spline_store_bind", s.store, gf.t, 0, 0, 1)
    fd.call("timefield3d_run", gf.t, p["dt"], p["steps"])
    o = _read(gf, s.mon, 1)[0]
    fd.call("fdtd_spline_store_unbind", s.store, gf.t)
    w = np.conj(o) / abs(o)
    fd.lib.timefield3d_zero_fields(ga.t)
    fd.call("timefield3d_set_exact_adjoint_schedule", ga.t, p["cx"], p["cy"], p["out_z"], s.mode.struct, 0, p["steps"],
            float(s.omega[0]), p["dt"], float(w.real), float(w.imag))
    fd.call("fdtd_spline_store_bind", s.store, ga.t, 1, p["steps"], -1)
    fd.call("timefield3d_run", ga.t, p["dt"], p["steps"] + 1)
    fd.call("fdtd_spline_store_unbind", s.store, ga.t)
    grad = np.zeros(NCTRL)
    cells = np.zeros(6 * (p["rows"][1] - p["rows"][0]) * (p["z1"] - p["z0"]))
    fd.call("fdtd_spline_store_gradient_exact", s.store, EP_CORE - EP_CLAD, _dptr(grad), _dptr(cells))
    return {"overlap": np.array([o]).astype(np.complex64), "gradient": grad.astype(np.float32),
            "cells": cells.astype(np.float32)}


def _run_sweep(s):
    grids = (fd.Timefield3d * len(s.sims))(*[g.t for g, _ in s.sims])
    steps = (C.c_int * len(s.sims))(*[p["steps"] for p in s.ps])
    for g, _ in s.sims:
        fd.lib.timefield3d_zero_fields(g.t)
    fd.call("fdtd_sweep_run", grids, len(s.sims), s.ps[0]["dt"], steps, 64, 0, 4.0)
    return np.stack([np.stack([_read(g, m, 11) for m in mons]) for g, mons in s.sims]).astype(np.complex64)


def _run_mode(s):
    s.libc.srand(s.seed & 0x7FFFFFFF)   # the solver starts from rand(), as the reference's does
    m, beta = s.modes.strip_mode(fd, s.case["mi"], s.case["mj"], 0.025, s.core, EP_CLAD, EP_CORE, LAM0,
                                 s.case["krylov"], s.case["tol"])
    return {"beta": np.array([beta]), "fields": m.fields}


def _run_train(s):
    s.net.set_params(s.w)
    loss = s.net.train(s.x, s.y, 1, batch=s.case["batch"], lr=3e-4, seed=1)
    return {"weights": s.net.get_params(), "loss": np.array([loss], np.float32)}


def _run_query(s):
    y = s.net.predict(s.x)
    dy = (2 * y / 11).astype(np.float32)   # of the mean transmission over 11 wavelengths
    return {"spectra": y, "gradient": s.net.input_gradient(s.x, dy)}


_RUN = {"run": _run_run, "dipole": _run_dipole, "driver": _run_driver, "adjoint": _run_adjoint, "sweep": _run_sweep,
        "mode": _run_mode, "train": _run_train, "query": _run_query}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _step_bytes(nx, ny, nz, L, value, lossy=False):
    """Fields read and written once, three E coefficients (six with loss), and the CPML auxiliaries in their slabs."""
    n = nx * ny * nz
    slabs = 2 * L * (ny * nz + nx * nz + nx * ny)
    return n * (12 * value + 4 * (6 if lossy else 3)) + slabs * 8 * value


def work(case):
    kind = case["kind"]
    if kind in ("run", "dipole", "driver", "adjoint"):
        nx, ny, nz = _dims(case)
        n, L = nx * ny * nz, case.get("cells", 0)
        value = 4 if case.get("precision") == "f32" or kind == "adjoint" else 8
        steps = case["steps"] * (2 if kind in ("driver", "adjoint") else 1)
        step = _step_bytes(nx, ny, nz, L, value, case.get("lossy", False))
        extra = n * 48 if case.get("fields") or kind == "driver" else 0
        if kind == "driver":
            extra += case["steps"] * nx * nz * 6 * 40   # the running DFT slice: read, accumulator read and written
        if kind == "adjoint":
            rows = 2 * max(2, min(4, ny // 16)) + 1
            extra += case["steps"] * 6 * rows * (nz - 2 * L - 36) * 3 * 4 * 4   # edge fields: stored and read, twice
        return {"bytes": step * steps + extra, "flops": 42.0 * n * steps}
    if kind == "sweep":
        cs = _sweep_cases(case, 0)
        return {"bytes": sum(c["steps"] * _step_bytes(c["nx"], c["ny"], c["nz"], 12, 4) for c in cs),
                "flops": sum(42.0 * c["steps"] * c["nx"] * c["ny"] * c["nz"] for c in cs)}
    if kind == "mode":
        # one Krylov cycle at the least: every basis vector written once and read once per orthogonalisation
        n, k = case["mi"] * case["mj"], case["krylov"]
        return {"bytes": n * (8 * 16 + 6 * 16) + n * 32 * k * (k + 1) / 2, "flops": n * (300.0 * k + 32.0 * k * (k + 1))}
    params = NCTRL * 256 + 2 * 256 * 256 + 256 * 22
    if kind == "train":
        steps = case["designs"] // case["batch"]
        return {"bytes": steps * (params * 4 * 7 + case["batch"] * 42 * 4), "flops": 6.0 * params * case["batch"] * steps}
    return {"bytes": params * 2 * 2 + case["rows"] * (NCTRL * 3 + 22 * 3) * 4, "flops": 6.0 * params * case["rows"]}


# ---------------------------------------------------------------------------
# the same results in 64 bits, plain torch
# ---------------------------------------------------------------------------
_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t64(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_DEV)


def _reduced(ph):
    """The phase modulo two of the reference's nine-digit pi, as its overlaps and DFTs take it."""
    return ph - int(ph / (2 * PI)) * 2 * PI


def _normalised(f, disc):
    p = np.sum(np.conj(f[..., 3]) * f[..., 1] - np.conj(f[..., 4]) * f[..., 0]
               + f[..., 3] * np.conj(f[..., 1]) - f[..., 4] * np.conj(f[..., 0]))
    return f / math.sqrt(abs(-0.5 * disc * disc * p))


class _Yee64:
    """Leapfrog in 64 bits on [z][y][x] tensors; interior update, then CPML terms inside it or the Mur faces after it."""

    def __init__(self, p, ep, sig, L):
        nx, ny, nz = p["nx"], p["ny"], p["nz"]
        self.dx, self.dt, self.L, self.N = p["dx"], p["dt"], L, (nx, ny, nz)
        self.ep = _t64(ep)
        self.F = [torch.zeros(nz, ny, nx, dtype=torch.float64, device=_DEV) for _ in range(6)]
        c = (slice(1, -1),) * 3
        s = _t64(sig)[c] if sig is not None else 0.0
        self.main = 1.0 / (self.ep[c] / self.dt + 0.5 * s)
        self.keep = self.ep[c] / self.dt - 0.5 * s
        self.src = {}                       # plane -> six [ny][nx] tensors
        if L:
            self.psi, self.tab = {}, {}
            for h in range(2):
                for a in range(3):
                    b, co = self._profile(self.N[a], L, h)
                    for side, at in ((0, slice(1, L)), (1, slice(self.N[a] - L, self.N[a] - 1))):
                        shape = [1, 1, 1]
                        shape[2 - a] = L - 1
                        self.tab[h, a, side] = _t64(b[at]).view(shape), _t64(co[at]).view(shape)
                        size = [nz - 2, ny - 2, nx - 2]
                        size[2 - a] = L - 1
                        for w in range(2):
                            self.psi[h, a, side, w] = torch.zeros(size, dtype=torch.float64, device=_DEV)

    def _profile(self, N, L, h):
        b, co = np.ones(N), np.zeros(N)
        smax = 0.8 * 4 / self.dx
        for i in range(N):
            q = i + 0.5 * h
            rho = (L - 0.5 - q) / L if q < L - 0.5 else (q - (N - L - 0.5)) / L if q > N - L - 0.5 else 0.0
            if rho > 0:
                s = smax * rho ** 3
                b[i] = math.exp(-s * self.dt)
                co[i] = b[i] - 1.0
        return b, co

    def _curl(self, h):
        """The curl of H (h = 0, backward differences) or E (h = 1, forward), interior, over dx."""
        o = 3 if h == 0 else 0
        c = slice(1, -1)
        n = slice(None, -2) if h == 0 else slice(2, None)

        def d(m, a):
            f = self.F[o + m]
            at = [c, c, c]
            at[2 - a] = n
            x = (f[c, c, c] - f[tuple(at)]) if h == 0 else (f[tuple(at)] - f[c, c, c])
            return x.div_(self.dx)
        D = {(m, a): d(m, a) for m, a in ((2, 1), (1, 2), (0, 2), (2, 0), (1, 0), (0, 1))}
        curl = [D[2, 1] - D[1, 2], D[0, 2] - D[2, 0], D[1, 0] - D[0, 1]]
        if self.L:
            for a, terms in ((0, ((1, 2, -1), (2, 1, 1))), (1, ((0, 2, 1), (2, 0, -1))), (2, ((0, 1, -1), (1, 0, 1)))):
                for side in range(2):
                    b, co = self.tab[h, a, side]
                    n0 = self.L - 1
                    start = 0 if side == 0 else D[1, 0].shape[2 - a] - n0
                    for w, (comp, m, sign) in enumerate(terms):
                        P = self.psi[h, a, side, w]
                        P.mul_(b).add_(D[m, a].narrow(2 - a, start, n0) * co)
                        curl[comp].narrow(2 - a, start, n0).add_(P, alpha=sign)
        return curl

    def _mur(self, old, efield):
        nx, ny, nz = self.N
        end = (nx, ny, nz)
        for high in range(2):
            for a in range(3):
                ib, ii = (end[a] - 1, end[a] - 2) if high else (0, 1)
                for c in range(3):
                    if c == a:
                        continue
                    m = c if efield else 3 + c
                    speed = self.dt / torch.sqrt(self.ep.select(2 - a, ib))
                    k = (speed - self.dx) / (speed + self.dx)
                    f = self.F[m]
                    f.select(2 - a, ib).copy_(old[m].select(2 - a, ii)
                                              + k * (f.select(2 - a, ii) - old[m].select(2 - a, ib)))

    def step(self):
        c = (slice(1, -1),) * 3
        old = None if self.L else [f.clone() for f in self.F]
        curl = self._curl(0)
        for z, J in self.src.items():
            for m in range(3):
                curl[m][z - 1] -= J[m][1:-1, 1:-1]
        for m in range(3):
            self.F[m][c] = self.main * (self.keep * self.F[m][c] + curl[m])
        if old:
            self._mur(old, 1)
        curl = self._curl(1)
        for z, J in self.src.items():
            for m in range(3):
                curl[m][z - 1] += J[3 + m][1:-1, 1:-1]
        for m in range(3):
            self.F[3 + m][c] -= self.dt * curl[m]
        if old:
            self._mur(old, 0)

    def set_source(self, z, planes):
        """Source planes are floats, as the reference's source array is."""
        self.src[z] = [v.to(torch.float32).to(torch.float64) for v in planes]

    def mode_source(self, z, e, phase, amp):
        c, s = math.cos(phase), math.sin(phase)
        ep = self.ep[z]
        w = [e[m].real * c + e[m].imag * s for m in range(6)]
        self.set_source(z, [amp * ep * w[m] for m in range(3)] + [amp * w[m] for m in range(3, 6)])

    def overlap(self, z, e, reverse=0):
        Ex, Ey, Hx, Hy = (self.F[m][z] for m in (0, 1, 3, 4))
        mHx, mHy = (-e[3].conj(), -e[4].conj()) if reverse else (e[3], e[4])
        return complex((Hx * e[1] - Hy * e[0] + Ey * mHx - Ex * mHy).sum()) * (-0.5 * self.dx * self.dx)


def _mode64(f, disc):
    f = _normalised(f, disc)
    return [torch.as_tensor(np.ascontiguousarray(f[..., m]), device=_DEV) for m in range(6)]


def _spline(K, n):
    """[n][K] weights of a natural cubic spline through K values placed evenly on 0..n-1."""
    h = (n - 1) / (K - 1)
    A = np.eye(K)
    B = np.zeros((K, K))
    for i in range(1, K - 1):
        A[i, i - 1:i + 2] = 1, 4, 1
        B[i, i - 1:i + 2] = 6 / h ** 2, -12 / h ** 2, 6 / h ** 2
    M = np.linalg.solve(A, B)
    z = np.arange(n)
    s = np.minimum((z / h).astype(int), K - 2)
    a, b = (z - s * h)[:, None], ((s + 1) * h - z)[:, None]
    I = np.eye(K)
    return M[s] * b ** 3 / (6 * h) + M[s + 1] * a ** 3 / (6 * h) + (I[s] / h - M[s] * h / 6) * b \
        + (I[s + 1] / h - M[s + 1] * h / 6) * a


def _taper_eps(p):
    """(eps [z][y][x], spline weights, left edges, right edges)"""
    clad, core = float(np.float32(EP_CLAD)), float(np.float32(EP_CORE))
    ep = np.full((p["nz"], p["ny"], p["nx"]), clad)
    b, t = p["rows"]
    ep[:p["z0"], b:t, p["w_in"][0]:p["w_in"][1]] = core
    ep[p["z1"]:, b:t, p["w_out"][0]:p["w_out"][1]] = core
    W = _spline(NCTRL, p["z1"] - p["z0"])
    half = (W @ p["widths"]) / (2 * p["dx"])
    i = np.arange(p["nx"])[None, :]
    f = np.minimum(i + 1.0, p["cx"] + half[:, None]) - np.maximum(i, p["cx"] - half[:, None])
    row = np.where(f >= 1, core, np.where(f > 0, (clad + f * (EP_CORE - clad)).astype(np.float32), clad))
    ep[p["z0"]:p["z1"], b:t] = row[:, None, :]
    return ep, W, p["cx"] - half, p["cx"] + half


def _sig(p):
    if not p["sig"]:
        return None
    s = np.zeros((p["nz"], p["ny"], p["nx"]))
    x0, x1, y0, y1, z0, z1 = p["sig_box"]
    s[z0:z1, y0:y1, x0:x1] = np.float32(p["sig"])
    return s


def _forward64(p, after=None):
    ep, _, _, _ = _taper_eps(p)
    y = _Yee64(p, ep, _sig(p), p["L"])
    ein, eout = _mode64(p["mode_in"], p["dx"]), _mode64(p["mode_out"], p["dx"])
    acc = np.zeros((2, len(p["omega"])), complex)
    for n in range(p["steps"]):
        y.mode_source(p["src_z"], ein, p["phase"][n], p["amp"][n])
        y.step()
        ph = np.exp([1j * _reduced(n * p["dt"] * w) for w in p["omega"]])
        acc += np.array([[y.overlap(p["launch_z"], ein)], [y.overlap(p["out_z"], eout)]]) * ph
        if after:
            after(y, n)
    return y, acc


def _stack(y):
    return torch.stack(y.F, dim=-1).cpu().numpy()


def _exact_run(case, seed):
    y, acc = _forward64(_taper(case, seed))
    return {"monitors": acc, "fields": _stack(y)} if case["fields"] else {"monitors": acc}


def _exact_dipole(case, seed):
    p = _dipole(case, seed)
    n = p["nx"]
    ep = np.ones((n, n, n))
    a, b = p["cube"]
    ep[a:b, a:b, a:b] = p["eps"]
    y = _Yee64(p, ep, None, 0)
    i, j, k = p["src"]
    J = [torch.zeros(n, n, dtype=torch.float64, device=_DEV) for _ in range(6)]
    y.src[k] = J
    out = torch.zeros(12, len(p["drive"]), dtype=torch.float64, device=_DEV)
    kk, jj, ii = (torch.tensor([pt[q] for pt in p["pts"]], device=_DEV) for q in (2, 1, 0))
    for s, v in enumerate(np.float32(p["drive"]).astype(float)):
        J[2][j, i] = v
        y.step()
        out[:, s] = torch.stack([y.F[m][kk, jj, ii] for m in range(3)], dim=1).reshape(-1)
    return out.cpu().numpy()


def _exact_driver(case, seed):
    p = _driver(case, seed)
    T, dt, b, t = p["T"], p["dt"], *p["rows"]
    ep = np.full((p["nz"], p["ny"], p["nx"]), float(np.float32(EP_CLAD)))
    core = float(np.float32(EP_CORE))
    ep[:p["z0"], b:t, p["wg_in"][0]:p["wg_in"][1]] = core
    ep[p["z1"]:, b:t, p["wg_out"][0]:p["wg_out"][1]] = core
    length, S = p["z1"] - p["z0"], p["seg"]
    ks, js, xs = [], [], []
    near = lambda v: math.floor(abs(v) + 0.5) * (1 if v >= 0 else -1)   # noqa: E731  C's round
    for n in range(S):
        s0, s1 = p["z0"] + n * length // S, p["z0"] + (n + 1) * length // S
        for k in range(s0, s1):
            edge = {e: (v[n], v[n + 1] - v[n]) for e, v in (("l", p["left"]), ("r", p["right"]))}
            lo, hi = (v + near(d / (s1 - s0) * (k - s0)) for v, d in (edge["l"], edge["r"]))
            ep[k, b:t, lo:hi] = core
            px = [v + int(d * (k - s0) / (s1 - s0)) for v, d in (edge["r"], edge["l"])]
            for j in range(b, t):
                ks += [k, k]
                js += [j, j]
                xs += px
    kk, jj, ii = (torch.tensor(v, device=_DEV) for v in (ks, js, xs))
    e = _mode64(p["mode"], p["dx"])
    y = _Yee64(p, ep, None, 0)
    cum = np.zeros(3, complex)
    four = torch.zeros(p["nz"], p["nx"], 6, dtype=torch.complex128, device=_DEV)
    fwd = []
    for n in range(T):
        phase = n * dt * p["omega"]
        y.mode_source(p["src_z"], e, phase, p["amp"][n])
        y.step()
        w = np.exp(1j * _reduced(phase))
        four += torch.stack([f[:, p["cy"]] for f in y.F], dim=-1) * complex(w)
        cum += w * np.array([y.overlap(p["launch_z"], e), y.overlap(p["launch_z"], e, 1), y.overlap(p["out_z"], e)])
        fwd.append(torch.stack([y.F[m][kk, jj, ii] for m in range(3)]))
    fields = _stack(y)
    y = _Yee64(p, ep, None, 0)
    grad = torch.zeros(len(ks), dtype=torch.float64, device=_DEV)
    zero = torch.zeros(p["ny"], p["nx"], dtype=torch.float64, device=_DEV)
    for n in range(T - 1, -1, -1):
        phase = (n + 1) * dt * p["omega"]
        w = [e[m].real * math.cos(phase) + e[m].imag * math.sin(phase) for m in range(6)]
        y.set_source(p["out_z"], [w[4], -w[3], zero, w[1], -w[0], zero])
        y.step()
        grad += sum(fwd[n][m] * y.F[m][kk, jj, ii] for m in range(3))
    return {"overlaps": cum, "fields": fields, "fourier": four.cpu().numpy(), "gradient": grad.cpu().numpy()}


def _exact_adjoint(case, seed):
    p = _taper(case, seed)
    p["omega"] = np.array([2 * PI / LAM0])
    T, (b, t) = p["steps"], p["rows"]
    ep, W, xl, xr = _taper_eps(p)
    height, length = t - b, p["z1"] - p["z0"]
    idx = [(int(min(max(math.floor(x[k]) + d, 0), p["nx"] - 1)), j, p["z0"] + k)
           for k in range(length) for j in range(b, t) for x in (xr, xl) for d in (-1, 0, 1)]
    ii, jj, kk = (torch.tensor([v[q] for v in idx], device=_DEV) for q in range(3))
    at = lambda y: torch.stack([y.F[m][kk, jj, ii] for m in range(3)])   # noqa: E731
    fwd = []
    _, acc = _forward64(p, lambda y, n: fwd.append(at(y)))
    o = acc[1, 0]
    w = np.conj(o) / abs(o)
    e = _mode64(p["mode_out"], p["dx"])
    y = _Yee64(p, ep, None, p["L"])
    grad = torch.zeros(len(idx), dtype=torch.float64, device=_DEV)
    zero = torch.zeros(p["ny"], p["nx"], dtype=torch.float64, device=_DEV)
    kappa = 0.5 * p["dx"] ** 2 / p["dt"]

    def drive(u):   # entry u of the schedule: Re(w m e^{i omega dt (T - u)}) of a mode component
        z = complex(w) * np.exp(1j * p["omega"][0] * p["dt"] * (T - u)) if 1 <= u <= T else 0.0
        return [kappa * (e[m] * z).real if z else zero for m in range(6)]
    for u in range(T + 1):
        J, M = drive(u), drive(u + 1)
        y.set_source(p["out_z"], [-J[4], J[3], zero, -M[1], M[0], zero])
        y.step()
        n = T - u
        if n < T:
            before = fwd[n - 1] if n > 0 else torch.zeros_like(fwd[0])
            grad -= (at(y) * (fwd[n] - before)).sum(dim=0)
    cells = grad.cpu().numpy()
    g = cells.reshape(length, height, 2, 3)[..., 1].sum(axis=(1, 2))
    return {"overlap": np.array([o]), "gradient": (W.T @ g) * (EP_CORE - EP_CLAD) / (2 * p["dx"]), "cells": cells}


def _exact_sweep(case, seed):
    return np.stack([_forward64(_taper(c, 100 * seed + i))[1] for i, c in enumerate(_sweep_cases(case, seed))])


def _layers(flat):
    out, o = [], 0
    w = _t64(flat)
    for n, i in ((256, NCTRL), (256, 256), (256, 256), (22, 256)):
        out += [w[o:o + n * i].reshape(n, i).clone().requires_grad_(), w[o + n * i:o + n * i + n].clone().requires_grad_()]
        o += n * i + n
    return out


def _net64(w, x):
    h = x
    for l in range(4):
        h = h @ w[2 * l].T + w[2 * l + 1]
        if l < 3:
            h = 0.5 * h * (1 + torch.erf(h / math.sqrt(2)))
    return h


def _exact_train(case, seed):
    x, y = (_t64(v) for v in _designs(case["designs"], seed + 1))
    w = _layers(_weights(seed))
    m, v = [torch.zeros_like(q) for q in w], [torch.zeros_like(q) for q in w]
    order = np.random.default_rng(1).permutation(len(x))
    bs = min(case["batch"], len(x) // 8 * 8)
    loss = None
    for k, s in enumerate(range(0, len(x) - bs + 1, bs), 1):
        at = torch.as_tensor(order[s:s + bs], device=_DEV)
        loss = ((_net64(w, x[at]) - y[at]) ** 2).mean()
        for q, (p, g) in enumerate(zip(w, torch.autograd.grad(loss, w))):
            m[q] = 0.9 * m[q] + 0.1 * g
            v[q] = 0.999 * v[q] + 0.001 * g * g
            p.data -= 3e-4 * (m[q] / (1 - 0.9 ** k)) / (torch.sqrt(v[q] / (1 - 0.999 ** k)) + 1e-8)
    return {"weights": torch.cat([q.detach().reshape(-1) for q in w]).cpu().numpy(), "loss": np.array([loss.item()])}


def _exact_query(case, seed):
    x = _t64(_designs(case["rows"], seed + 1)[0]).requires_grad_()
    y = _net64(_layers(_weights(seed)), x)
    g, = torch.autograd.grad(y, x, 2 * y.detach() / 11)
    return {"spectra": y.detach().cpu().numpy(), "gradient": g.cpu().numpy()}


_EXACT = {"run": _exact_run, "dipole": _exact_dipole, "driver": _exact_driver, "adjoint": _exact_adjoint,
          "sweep": _exact_sweep, "train": _exact_train, "query": _exact_query}


def exact(case, seed):
    # a mode is defined by its solver's start vector and stopping rule, so it has no value of its own in 64 bits
    return _EXACT[case["kind"]](case, seed) if case["kind"] in _EXACT else None
