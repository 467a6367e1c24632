// tile_cells.cuh -- one tile (band of rows x range of columns x chunk of planes)
// of the one-pass FP32 Yee step with one E coefficient a cell, by a thread block
// (yee_tile.cu has the design, the launches and the plan).
#pragma once

#include "stream_cells.cuh"

#include <type_traits>

namespace fdtd {

// Shared memory of a block: slot p = row * sw + quad (sw: left halo, owned quads,
// right halo; a tile at a row's end has no halo there) of every staged array, an
// array's slots together and kSlots apart, so a thread's own quad of every array is
// one pointer and a constant, and a plane's rows of an array are one TMA box (cells
// outside the grid read 0).  The H arrays start one row lower than the others: E's
// update reads H of row j - 1.
template <bool LOSSY> struct TileMem {
    static constexpr int kSlots = LOSSY ? 448 : 480;         // (tp + 1) * sw at most
    static constexpr int kArr = 4 * kSlots;                  // floats between arrays
    static constexpr int kArrays = LOSSY ? 8 : 7;            // Hx Hy Hz Ex Ey Ez cb (ca)
    static constexpr int kStage = kArrays * kArr;
    static constexpr int kENew = 3 * kArr;
};
constexpr int kTileMaxQuads = 64;   // a row of a box: 256 cells

struct TileShape {                // of a block's shared memory
    int tp, sw;                   // staged rows; slots a row
    __host__ __device__ int xpsi(int L) const { return L > 0 ? 4 * tp * stream_xpsi_stride(L) : 0; }
    __host__ __device__ size_t floats(bool lossy, int L) const
    {
        const size_t arrays = lossy ? (size_t)kStreamStages * TileMem<true>::kStage + 2 * TileMem<true>::kENew
                                    : (size_t)kStreamStages * TileMem<false>::kStage + 2 * TileMem<false>::kENew;
        // (8 more: the last slot's right neighbour is read, and not used, past the arrays)
        return arrays + (size_t)kStreamStages * xpsi(L) + (L > 0 ? 36 * (size_t)L : 0) + 8;
    }
    __host__ __device__ bool fits(bool lossy) const
    {
        return sw <= kTileMaxQuads && (tp + 1) * sw <= (lossy ? TileMem<true>::kSlots : TileMem<false>::kSlots);
    }
};

// Thread roles of a tile of quads [q0, q1): threads of interior quads (and of the
// right halo quad, when the tile ends inside the row), row by row; then, in warps
// of their own, one thread a cell of the tile's x-slab quads.
struct TileRoles {
    int qa, qb;      // interior quads [qa, qb) of the tile
    int halo;        // 1: quad q1 is computed too (its new E is the +x neighbour's)
    int nl, nr;      // x-slab quads at the left and right end
    int xbase;       // first thread of the x-cell warps
    int threads;
};

__host__ __device__ inline TileRoles tile_roles(int nx, int L, int q0, int q1, int tp)
{
    const int QX = nx / 4;
    int QL = 0, QR = QX;
    if (L > 0) {
        QL = (L + 3) / 4;
        QR = (nx - L) / 4;
        if (QR < QL) QR = QL;
        if (QR > QX) QR = QX;
    }
    TileRoles r{};
    r.qa = q0 > QL ? q0 : (QL < q1 ? QL : q1);
    r.qb = q1 < QR ? q1 : (QR > r.qa ? QR : r.qa);
    r.halo = q1 < QX ? 1 : 0;
    r.nl = r.qa - q0;
    r.nr = q1 - r.qb;
    r.xbase = (tp * (r.qb - r.qa + r.halo) + 31) / 32 * 32;
    r.threads = (r.xbase + tp * 4 * (r.nl + r.nr) + 31) / 32 * 32;
    return r;
}

// the plane's barrier of the tile's `n` threads (whole warps; both kinds meet here)
__device__ __forceinline__ void tile_barrier(int n) { asm volatile("bar.sync 1, %0;\n" ::"r"(n) : "memory"); }

__device__ __forceinline__ unsigned tile_s32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

// Barriers of the staged planes.  A wait is bounded (kTileWaitNs): one that gives
// up sets the abort flag, which every later wait sees, and the tile runs on
// without waiting to its end, so all threads still meet at its barriers; the
// caller's *err reports it.
struct TileSync {
    unsigned long long full[kStreamStages];   // plane m = it + 1 has landed in stage m % 3
    int abort;
};

__device__ __forceinline__ void tile_sync_init(TileSync *y)
{
    if (threadIdx.x != 0) return;
    for (int q = 0; q < kStreamStages; q++)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"((unsigned)__cvta_generic_to_shared(&y->full[q])));
    y->abort = 0;
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
}
constexpr unsigned long long kTileWaitNs = 1000000000ull;

__device__ __forceinline__ bool tile_wait(TileSync *y, unsigned long long *bar, unsigned parity, bool after_abort = false,
                                          unsigned long long limit_ns = kTileWaitNs)
{
    const unsigned a = tile_s32(bar);
    unsigned long long t0 = 0;
    for (;;) {
        unsigned ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(ok)
                     : "r"(a), "r"(parity)
                     : "memory");
        if (ok) return true;
        if (!after_abort && *(volatile int *)&y->abort) return false;
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        if (!t0) t0 = now;
        else if (now - t0 > limit_ns) {
            y->abort = 1;
            return false;
        }
    }
}

// one box of a plane (x, y: its first cell, x a multiple of 4) that counts on mbarrier `bar`
__device__ __forceinline__ void tile_box(float *dst, const CUtensorMap *map, int x, int y, int z, unsigned long long *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];\n" ::"r"(tile_s32(dst)),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(tile_s32(bar))
        : "memory");
}

// Iteration it (plane k = k0 + it, it = 0..n) updates E of plane k on the owned
// rows, the halo row j0 + rows and the right halo quad, and H of plane k - 1 on
// the owned rows.  Plane k sits in stage it % 3; right after the plane's barrier
// the stage of plane k - 1 takes the copies of plane k + 2.
//
// Quad threads keep the old H and the new E of their quad in plane k - 1 in
// registers on planes outside the z slabs (rows outside the y slabs); where a
// cell carries y or z auxiliaries both come from shared memory instead, since
// the auxiliaries of the next plane, loaded an iteration ahead, need the
// registers.  The two kinds of planes are loops of their own, so neither holds
// the other's state.
//
// before(): run by all threads before the copies of the first planes; during(): while
// they are on their way.
template <bool CPML, bool LOSSY, typename Before, typename During>
__device__ __forceinline__ void yee_tile(const StreamArgs &a, const TileMaps *maps, const TileBox tl,
                                         const TileShape sh, float *sm, TileSync *sync, int *err, Before before,
                                         During during)
{
    constexpr int S = kStreamStages;
    const int nx = a.nx, ny = a.ny, nz = a.nz, L = CPML ? a.L : 0;
    const int TP = sh.tp, SW = sh.sw, R = tl.rows, QX = nx >> 2;
    const int XW = stream_xpsi_stride(L);
    const sidx_t nxy = (sidx_t)nx * (sidx_t)ny;
    const TileRoles ro = tile_roles(nx, L, tl.q0, tl.q1, TP);
    const int tid = (int)threadIdx.x;
    const int n = tl.k1 - tl.k0;
    const float dx = a.dx, div = 1.0f / dx, hb = a.hb;
    using M = TileMem<LOSSY>;
    constexpr int A = M::kArr;
    const int row_st = 4 * SW;
    const int xp_st = sh.xpsi(L);
    float *stage = sm;                                   // [S][arrays][slots]
    float *enew = stage + S * M::kStage;                 // [2][Ex Ey Ez][slots]
    float *xps = enew + 2 * M::kENew;                    // [S][4][TP][XW]
    float *ptab = xps + S * xp_st;
    if (CPML) stream_profile_table(ptab, a);
    const int NT = ro.threads;
    before();
    // thread 0 copies: one TMA box a plane and array.  Plane it + 2 goes into the
    // stage of plane it - 1 right after the barrier of iteration it, when every
    // thread is done with iteration it - 1.
    auto copy = [&](int it, bool h_only) {
        const int m = it + 1, k = tl.k0 + it, x = 4 * (tl.q0 - (tl.q0 > 0 ? 1 : 0));
        const unsigned h_bytes = 3u * 16u * (unsigned)((TP + 1) * SW);
        const unsigned all_bytes = h_bytes + (unsigned)(M::kArrays - 3) * 16u * (unsigned)(TP * SW);
        unsigned long long *bar = &sync->full[m % S];
        float *st = stage + (m % S) * M::kStage;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(tile_s32(bar)),
                     "r"(h_only ? h_bytes : all_bytes)
                     : "memory");
#pragma unroll
        for (int c = 0; c < 3; c++) tile_box(st + c * A, &maps->h[c], x, tl.j0 - 1, k, bar);
        if (h_only) return;
#pragma unroll
        for (int c = 0; c < 3; c++) tile_box(st + (3 + c) * A, &maps->e[c], x, tl.j0, k, bar);
        tile_box(st + 6 * A, &maps->cb, x, tl.j0, k, bar);
        if (LOSSY) tile_box(st + 7 * A, &maps->ca, x, tl.j0, k, bar);
    };
    if (tid == 0) {
        copy(-1, true);
        copy(0, false);
        copy(1, false);      // a tile has at least one plane
    }
    during();
    __syncthreads();
    if (tid >= NT) return;
    auto wait_plane = [&](int it) {
        const int m = it + 1;
        tile_wait(sync, &sync->full[m % S], (unsigned)(m / S) & 1u);
    };
    // start of iteration it: plane it has landed, the new E of plane it - 1 is there
    auto begin = [&](int it) {
        wait_plane(it);
        tile_barrier(NT);
        if (tid == 0 && it + 2 <= n) copy(it + 2, false);
    };
    // a wait gave up: report it, and let the copies in flight land (with a limit)
    auto finish = [&]() {
        if (tid != 0 || !*(volatile int *)&sync->abort) return;
        atomicExch(err, 1);
        for (int m = n + 1; m >= 0 && m > n + 1 - S; m--) tile_wait(sync, &sync->full[m % S], (unsigned)(m / S) & 1u, true);
    };
    auto z_plane = [&](int k) { return CPML && (k < L || k >= nz - L); };

    if (!CPML || tid < ro.xbase) {
        // ---- interior quads and the right halo quad; r = TP: idle
        const int QW = ro.qb - ro.qa + ro.halo;
        const int r = QW > 0 && tid < TP * QW ? tid / QW : TP;
        const int v = r < TP ? tid - r * QW : 0;
        const int q = v < ro.qb - ro.qa ? ro.qa + v : tl.q1;
        const bool right = ro.halo && q == tl.q1;        // computed for its neighbour only
        const bool act = right ? r < R : r <= R;
        const bool own = r < R && !right;
        const int j = tl.j0 + r, i0 = 4 * q, lq = q - tl.q0 + (tl.q0 > 0 ? 1 : 0);
        const sidx_t ij0 = (sidx_t)i0 + (sidx_t)nx * (sidx_t)j;
        const bool row_upd = j >= 1 && j <= ny - 2;      // false only for a halo row on the shell
        const bool y_row = CPML && (j < L || j >= ny - L);
        auto yz_plane = [&](int k) { return y_row || z_plane(k); };
        const int slot = act ? 4 * (r * SW + lq) : 0;
        // E of plane k from the staged records; e: the quad's old, then new E
        struct Staged { Vf<4> hx, hy, hz, hxj, hzj, b, c; float hyi, hzi; };
        auto staged = [&](int s, Staged &t, Vf<4> (&e)[3]) {
            const float *rec = stage + s * M::kStage + slot;
            const float *hr = rec + row_st;
            t.hx = lds4(hr); t.hy = lds4(hr + A); t.hz = lds4(hr + 2 * A);
            e[0] = lds4(rec + 3 * A); e[1] = lds4(rec + 4 * A); e[2] = lds4(rec + 5 * A);
            t.b = lds4(rec + 6 * A);
            if (LOSSY) t.c = lds4(rec + 7 * A);
            else t.c = fillv<4>(1.f);
            t.hxj = lds4(rec); t.hzj = lds4(rec + 2 * A);
            t.hyi = hr[A - 1];            // left neighbour's last Hy, Hz (unused at x = 0)
            t.hzi = hr[2 * A - 1];
        };
        auto put_e = [&](int it, const Vf<4> (&e)[3]) {
            float *p = enew + (it & 1) * M::kENew + slot;
            sts4(p, e[0]); sts4(p + A, e[1]); sts4(p + 2 * A, e[2]);
        };
        auto store3 = [&](int f, int k, const Vf<4> (&x)[3]) {
            const sidx_t g = ij0 + nxy * (sidx_t)k;
#pragma unroll
            for (int c = 0; c < 3; c++) stv<4>(a.f_out[f + c] + g, x[c]);
        };
        const bool lo_end = !CPML && q == 0, hi_end = !CPML && q == QX - 1;   // x = 0, x = nx-1 stay

        // old H of the quad in the plane below, kept from one iteration to the next
        Vf<4> hp[3];
#pragma unroll
        for (int c = 0; c < 3; c++) hp[c] = fillv<4>(0.f);
        auto below = [&]() {   // iteration 0: of the plane below the tile (its stage is refilled after the barrier)
            wait_plane(-1);
            const float *rec = stage + slot + row_st;
#pragma unroll
            for (int c = 0; c < 3; c++) hp[c] = lds4(rec + c * A);
        };

        // planes with no y- or z-slab cell in this thread's E(k) and H(k-1)
        auto plain = [&](int it0, int it1) {
            Vf<4> ep[3];
#pragma unroll
            for (int c = 0; c < 3; c++) ep[c] = fillv<4>(0.f);
            for (int it = it0; it < it1; it++) {
                const int k = tl.k0 + it, s = (it + 1) % S;
                if (it == 0) below();
                begin(it);
                if (it == it0 && it > 0) {   // the other loop left the new E of the plane below in shared memory
                    const float *pe = enew + ((it - 1) & 1) * M::kENew + slot;
#pragma unroll
                    for (int c = 0; c < 3; c++) ep[c] = lds4(pe + c * A);
                }
                if (!act) continue;
                Staged t;
                Vf<4> e[3];
                staged(s, t, e);
                const float *sp = a.src.n ? src_plane(a.src, k) : nullptr;
                if (row_upd && k <= nz - 2) {
                    const Vf<4> e_old0 = e[0], e_old1 = e[1], e_old2 = e[2];
#pragma unroll
                    for (int x = 0; x < 4; x++) {
                        const float hyi = x == 0 ? t.hyi : t.hy.v[x - 1], hzi = x == 0 ? t.hzi : t.hz.v[x - 1];
                        float cx = (t.hz.v[x] - t.hzj.v[x]) - (t.hy.v[x] - hp[1].v[x]);
                        float cy = (t.hx.v[x] - hp[0].v[x]) - (t.hz.v[x] - hzi);
                        float cz = (t.hy.v[x] - hyi) - (t.hx.v[x] - t.hxj.v[x]);
                        if (sp) {
                            cx -= dx * sp[ij0 + x];
                            cy -= dx * sp[nxy + ij0 + x];
                            cz -= dx * sp[2 * nxy + ij0 + x];
                        }
                        e[0].v[x] = t.c.v[x] * e[0].v[x] + t.b.v[x] * cx;
                        e[1].v[x] = t.c.v[x] * e[1].v[x] + t.b.v[x] * cy;
                        e[2].v[x] = t.c.v[x] * e[2].v[x] + t.b.v[x] * cz;
                    }
                    if (lo_end) { e[0].v[0] = e_old0.v[0]; e[1].v[0] = e_old1.v[0]; e[2].v[0] = e_old2.v[0]; }
                    if (hi_end) { e[0].v[3] = e_old0.v[3]; e[1].v[3] = e_old1.v[3]; e[2].v[3] = e_old2.v[3]; }
                }
                put_e(it, e);
                if (own) {
                    if (it < n) store3(0, k, e);
                    if (it >= 1) {
                        const int km = k - 1;
                        const float *pe = enew + ((it - 1) & 1) * M::kENew + slot;
                        const Vf<4> exj = lds4(pe + row_st), ezj = lds4(pe + row_st + 2 * A);
                        const float eyr = pe[A + 4], ezr = pe[2 * A + 4];
                        const float *sph = a.src.n ? src_plane(a.src, km) : nullptr;
                        Vf<4> h[3];
#pragma unroll
                        for (int x = 0; x < 4; x++) {
                            const float eyi = x == 3 ? eyr : ep[1].v[x == 3 ? 3 : x + 1];
                            const float ezi = x == 3 ? ezr : ep[2].v[x == 3 ? 3 : x + 1];
                            float cx = (ezj.v[x] - ep[2].v[x]) - (e[1].v[x] - ep[1].v[x]);
                            float cy = (e[0].v[x] - ep[0].v[x]) - (ezi - ep[2].v[x]);
                            float cz = (eyi - ep[1].v[x]) - (exj.v[x] - ep[0].v[x]);
                            if (sph) {
                                cx += dx * sph[3 * nxy + ij0 + x];
                                cy += dx * sph[4 * nxy + ij0 + x];
                                cz += dx * sph[5 * nxy + ij0 + x];
                            }
                            h[0].v[x] = hp[0].v[x] - hb * cx;
                            h[1].v[x] = hp[1].v[x] - hb * cy;
                            h[2].v[x] = hp[2].v[x] - hb * cz;
                        }
                        if (lo_end) { h[0].v[0] = hp[0].v[0]; h[1].v[0] = hp[1].v[0]; h[2].v[0] = hp[2].v[0]; }
                        if (hi_end) { h[0].v[3] = hp[0].v[3]; h[1].v[3] = hp[1].v[3]; h[2].v[3] = hp[2].v[3]; }
                        store3(3, km, h);
                    }
                }
                hp[0] = t.hx; hp[1] = t.hy; hp[2] = t.hz;
                ep[0] = e[0]; ep[1] = e[1]; ep[2] = e[2];
            }
        };

        // planes with y- or z-slab cells (Y, Z: of which slabs).  With one kind the
        // auxiliaries of the next iteration are on their way during this one; with
        // both their registers do not suffice, and they are loaded at its end.
        auto slabs = [&](auto yc, auto zc, int it0, int it1) {
            constexpr bool Y = decltype(yc)::value, Z = decltype(zc)::value, AHEAD = !(Y && Z);
            YZPsi<4> yze, yzh;
            XPsi<4> xnone;
#pragma unroll
            for (int e = 0; e < 4; e++) { xnone.valid[e] = false; xnone.p0[e] = xnone.p1[e] = 0.f; }
            auto load1 = [&](YZPsi<4> &p, auto a0, bool any, int k) {
                constexpr int A0 = decltype(a0)::value;
                p.sj = Y && any ? slab_local(j, ny, L) : -1;
                p.sk = Z && any ? slab_local(k, nz, L) : -1;
                p.pxy = fillv<4>(0.f); p.pzy = p.pxy; p.pxz = p.pxy; p.pyz = p.pxy;
                if (Y && p.sj >= 0) {
                    const sidx_t sy = (sidx_t)i0 + (sidx_t)nx * (sidx_t)(p.sj + 2 * L * k);
                    p.pxy = ldv_rw<4>(a.psi_in[1][A0] + sy);
                    p.pzy = ldv_rw<4>(a.psi_in[1][A0 + 1] + sy);
                }
                if (Z && p.sk >= 0) {
                    const sidx_t sz = ij0 + nxy * (sidx_t)p.sk;
                    p.pxz = ldv_rw<4>(a.psi_in[2][A0] + sz);
                    p.pyz = ldv_rw<4>(a.psi_in[2][A0 + 1] + sz);
                }
                if (!Y) p.sj = -1;
                if (!Z) p.sk = -1;
            };
            auto load_yz = [&](YZPsi<4> &pe, YZPsi<4> &ph, int it) {
                const int k = tl.k0 + it;
                load1(pe, std::integral_constant<int, 0>{}, it < it1 && act && row_upd && k <= nz - 2, k);
                load1(ph, std::integral_constant<int, 2>{}, it < it1 && own && it >= 1, k - 1);
            };
            load_yz(yze, yzh, it0);
            for (int it = it0; it < it1; it++) {
                const int k = tl.k0 + it, s = (it + 1) % S;
                if (it == 0) below();
                // before the barrier: on their way while the block's warps meet (after it a
                // 200x160x400 step takes 160.7 us, 158.0 so; 256x128x128 70.2 and 68.3)
                YZPsi<4> ne, nh;
                if constexpr (AHEAD) load_yz(ne, nh, it + 1);
                begin(it);
                if (!act) continue;
                Vf<4> e[3];
                {
                    Staged t;
                    staged(s, t, e);
                    if (row_upd && k <= nz - 2) {
                        const float *sp = a.src.n ? src_plane(a.src, k) : nullptr;
                        stream_e_group<4, false, false, true, LOSSY>(
                            e[0], e[1], e[2], t.hx, t.hy, t.hz, hp[0], hp[1], t.hxj, t.hzj, t.hyi, t.hzi, t.b, t.b,
                            t.b, t.c, t.c, t.c, xnone, yze, ptab, a, i0, sp, ij0, nxy, dx, div);
                    }
                }
                put_e(it, e);
                if (own) {
                    if (it < n) {
                        store3(0, k, e);
                        if (yz_plane(k)) stream_psi_store<4, 0, false>(xnone, yze, a, i0, j, k, ij0, nxy);
                    }
                    if (it >= 1) {
                        const int km = k - 1;
                        const float *pe = enew + ((it - 1) & 1) * M::kENew + slot;
                        const Vf<4> ep0 = lds4(pe), ep1 = lds4(pe + A), ep2 = lds4(pe + 2 * A);
                        const Vf<4> exj = lds4(pe + row_st), ezj = lds4(pe + row_st + 2 * A);
                        const float *sp = a.src.n ? src_plane(a.src, km) : nullptr;
                        stream_h_group<4, false, false, true>(hp[0], hp[1], hp[2], e[0], e[1], ep0, ep1, ep2, exj,
                                                                     ezj, pe[A + 4], pe[2 * A + 4], xnone,
                                                                     yzh, ptab, a, i0, sp, ij0, nxy, dx, div, hb);
                        store3(3, km, hp);
                        if (yz_plane(km)) stream_psi_store<4, 2, false>(xnone, yzh, a, i0, j, km, ij0, nxy);
                    }
                }
                const float *rec = stage + s * M::kStage + slot + row_st;
#pragma unroll
                for (int c = 0; c < 3; c++) hp[c] = lds4(rec + c * A);
                if constexpr (AHEAD) { yze = ne; yzh = nh; }
                else load_yz(yze, yzh, it + 1);
            }
        };
        if constexpr (CPML) {
            // a warp's threads change loops together: by the band's rows, not the thread's
            const bool y_band = tl.j0 < L || tl.j0 + R >= ny - L;
            // iterations whose E(k) and H(k-1) lie in planes [L, nz - L)
            int a0 = L + 1 - tl.k0, a1 = nz - L - tl.k0;
            if (tl.k0 == L) a0 = 0;   // H(k0 - 1) is not this tile's
            a0 = a0 < 0 ? 0 : (a0 > n + 1 ? n + 1 : a0);
            a1 = a1 < a0 ? a0 : (a1 > n + 1 ? n + 1 : a1);
            const std::true_type yes;
            const std::false_type no;
            if (y_band) {
                if (a0 > 0) slabs(yes, yes, 0, a0);
                if (a1 > a0) slabs(yes, no, a0, a1);
                if (a1 < n + 1) slabs(yes, yes, a1, n + 1);
            } else {
                if (a0 > 0) slabs(no, yes, 0, a0);
                if (a1 > a0) plain(a0, a1);
                if (a1 < n + 1) slabs(no, yes, a1, n + 1);
            }
        } else {
            plain(0, n + 1);
        }
        finish();
        return;
    }
    if constexpr (CPML) {
        // ---- x-slab cells, one per thread; the 4 lanes of a quad are consecutive
        //      and share the 16-byte copies of its auxiliaries (lane e moves
        //      auxiliary e, two planes ahead, into a ring like the planes'); r = TP: idle
        const int NXC = 4 * (ro.nl + ro.nr);
        const int u = tid - ro.xbase;
        const int r = u < TP * NXC ? u / NXC : TP;
        const int cc = r < TP ? u - r * NXC : 0;
        const int v = cc >> 2, e4 = cc & 3;
        const int q = v < ro.nl ? tl.q0 + v : ro.qb + (v - ro.nl);
        const int i0 = 4 * q, i = i0 + e4, lq = q - tl.q0 + (tl.q0 > 0 ? 1 : 0);
        const bool act = r <= R;
        const bool own = r < R;
        const int j = tl.j0 + r;
        const sidx_t ijq = (sidx_t)i0 + (sidx_t)nx * (sidx_t)j;   // the quad's first cell
        const sidx_t ij = ijq + (sidx_t)e4;                       // this thread's cell
        const bool row_upd = j >= 1 && j <= ny - 2;
        const bool y_row = j < L || j >= ny - L;
        auto yz_plane = [&](int k) { return y_row || z_plane(k); };
        const bool whole = xquad_whole(i0, nx, L);
        const int si = slab_local(i, nx, L);
        const bool xvalid = si >= 0 && i >= 1 && i <= nx - 2;   // x terms updated at this cell
        const int slot = act ? 4 * (r * SW + lq) : 0;
        const int xslot = act ? r * XW : 0;
        float pxe[3] = {0.f, 0.f, 1.f}, pxh[3] = {0.f, 0.f, 1.f};
        if (xvalid) {
#pragma unroll
            for (int w = 0; w < 3; w++) {
                pxe[w] = __ldg(a.prof[w][0] + i);
                pxh[w] = __ldg(a.prof[3 + w][0] + i);
            }
        }
        // x-slab auxiliaries of iteration `it` into slot (it + S) % S, one group per call
        const float *psrc = a.psi_in[0][e4];
        auto issue = [&](int it) {
            if (it <= n && act) {
                const int k = tl.k0 + it;
                const sidx_t xs0 = (sidx_t)(2 * L) * ((sidx_t)j + (sidx_t)ny * (sidx_t)k);
                float *xr = xps + ((it + S) % S) * xp_st + xslot;
                if (whole) {
                    const int si0 = slab_local(i0, nx, L);
                    cp_async16(xr + e4 * TP * XW + si0, psrc + xs0 + si0);
                } else if (si >= 0) {
#pragma unroll
                    for (int arr = 0; arr < 4; arr++) cp_async4(xr + arr * TP * XW + si, a.psi_in[0][arr] + xs0 + si);
                }
            }
            cp_async_commit_group();
        };
        issue(0);
        issue(1);
        YZPsi<1> yze, yzh;
        auto load_yz = [&](int it) {
            yze.sj = yze.sk = yzh.sj = yzh.sk = -1;
            if (it > n) return;
            const int k = tl.k0 + it;
            if (!yz_plane(k) && !yz_plane(k - 1)) return;
            if (act && row_upd && k <= nz - 2) stream_yzpsi_load<1, 0>(yze, a, i, j, k, ij, nxy, ptab);
            if (own && it >= 1) stream_yzpsi_load<1, 2>(yzh, a, i, j, k - 1, ij, nxy, ptab);
        };
        load_yz(0);
        Vf<1> hxm = fillv<1>(0.f), hym = hxm, hzm = hxm;           // old H of the cell in the plane below
        for (int it = 0; it <= n; it++) {
            const int k = tl.k0 + it;
            const int s = (it + 1) % S;                       // this plane's stage
            const int xs = it % S, xp = (it + S - 1) % S;          // auxiliaries of this plane, of the plane below
            const bool e_upd = act && row_upd && k <= nz - 2;
            const bool h_upd = own && it >= 1;
            cp_async_wait_group<1>();
            if (it == 0) {
                wait_plane(-1);
                const float *rp = stage + slot + row_st + e4;
                hxm.v[0] = rp[0];
                hym.v[0] = rp[A];
                hzm.v[0] = rp[2 * A];
            }
            begin(it);
            // H's x-slab auxiliaries of the plane below; every lane of the quad
            // reads before any refills them
            XPsi<1> xsh;
            const float *xq = xps + xp * xp_st + xslot;
            stream_xpsi_cell(xsh, xq + 2 * TP * XW, xq + 3 * TP * XW, si, h_upd && xvalid, pxh);
            __syncwarp();
            issue(it + 2);

            const float *rec = stage + s * M::kStage + slot + e4;
            Vf<1> ex, ey, ez;
            ex.v[0] = rec[3 * A];
            ey.v[0] = rec[4 * A];
            ez.v[0] = rec[5 * A];
            XPsi<1> xse;
            const float *xr = xps + xs * xp_st + xslot;
            stream_xpsi_cell(xse, xr, xr + TP * XW, si, e_upd && xvalid, pxe);
            if (e_upd) {
                Vf<1> hx, hy, hz, hxj, hzj, b, c = fillv<1>(1.f);
                const float *hr = rec + row_st;
                hx.v[0] = hr[0];
                hy.v[0] = hr[A];
                hz.v[0] = hr[2 * A];
                hxj.v[0] = rec[0];
                hzj.v[0] = rec[2 * A];
                const float hyi = hr[A - 1], hzi = hr[2 * A - 1];   // unused at x = 0
                b.v[0] = rec[6 * A];
                if (LOSSY) c.v[0] = rec[7 * A];
                const float *sp = a.src.n ? src_plane(a.src, k) : nullptr;
                stream_e_group<1, true, true, true, LOSSY>(ex, ey, ez, hx, hy, hz, hxm, hym, hxj, hzj, hyi, hzi,
                                                                  b, b, b, c, c, c, xse, yze, ptab, a, i, sp, ij, nxy,
                                                                  dx, div);
            }
            if (act) {
                float *p = enew + (it & 1) * M::kENew + slot + e4;
                p[0] = ex.v[0];
                p[A] = ey.v[0];
                p[2 * A] = ez.v[0];
            }
            if (own && it < n) {
                const sidx_t g = ij + nxy * (sidx_t)k;
                a.f_out[0][g] = ex.v[0];
                a.f_out[1][g] = ey.v[0];
                a.f_out[2][g] = ez.v[0];
                stream_psi_store<1, 0, true>(xse, yze, a, i, j, k, ij, nxy);
            }
            if (h_upd) {
                const int km = k - 1;
                const float *pe = enew + ((it - 1) & 1) * M::kENew + slot + e4;
                Vf<1> exm, eym, ezm, exj, ezj;
                exm.v[0] = pe[0];
                eym.v[0] = pe[A];
                ezm.v[0] = pe[2 * A];
                exj.v[0] = pe[row_st];
                ezj.v[0] = pe[row_st + 2 * A];
                const float *sp = a.src.n ? src_plane(a.src, km) : nullptr;
                stream_h_group<1, true, true, true>(hxm, hym, hzm, ex, ey, exm, eym, ezm, exj, ezj, pe[A + 1], pe[2 * A + 1],
                                                           xsh, yzh, ptab, a, i, sp, ij, nxy, dx, div, hb);
                const sidx_t g = ij + nxy * (sidx_t)km;
                a.f_out[3][g] = hxm.v[0];
                a.f_out[4][g] = hym.v[0];
                a.f_out[5][g] = hzm.v[0];
                stream_psi_store<1, 2, true>(xsh, yzh, a, i, j, km, ij, nxy);
            }
            const float *hr = rec + row_st;
            hxm.v[0] = hr[0];
            hym.v[0] = hr[A];
            hzm.v[0] = hr[2 * A];
            load_yz(it + 1);
        }
        cp_async_wait_group<0>();
        finish();
    }
}

}  // namespace fdtd
