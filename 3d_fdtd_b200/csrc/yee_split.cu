// yee_split.cu -- separate E and H passes and the Mur boundary.
//
// This is the path that reproduces the reference step
// timefield3d_apply_timestep_omp_full (timefield3d.c:2787-2849) exactly:
//   shell snapshot -> E interior -> E Mur faces -> H interior -> H Mur faces.
// In FP64 every interior and boundary value is bit-identical to the
// reference's (same operations, same order, no FMA).  It also carries the
// CPML terms for grids that use FP64 or the non-fused FP32 path.
//
// Thread layout: one thread a cell, a block 256 consecutive cells of a plane
// (x fastest), every load of a cell issued before its arithmetic and its
// stores.  Both updates are bound by memory: E reads E, H and ep and writes E (84
// B a cell in FP64), H reads both and writes H (72 B).  A thread used to walk
// 16 planes to keep the z neighbour in a register; its loads then waited for the
// previous plane's stores (the arrays may alias), one memory latency a plane,
// and a 64^3 grid had 128 blocks.  With a thread a cell the z and y neighbours
// come from L2: FP64 steps of the 200 x 160 x 400 grid with a 12-cell CPML went
// from 0.85 to 0.48 ms (the cells in no slab move 4.8 TB/s in E, 5.9 in H, the slabs' 3.7 and 3.9), and of
// a 64^3 grid with the Mur boundary from 104 to 25 us (18 now).
// FP64 divisions cost as much as a third of the traffic: a cell whose three
// permittivities are equal (every rasteriser writes them so) takes its
// coefficient once (and reads one, where that holds for every cell of the grid; with H
// going backwards over the blocks, to start on what E left in L2: 483 to 473 us).
#include "common.cuh"
#include "kernels.h"

#include <algorithm>

namespace fdtd {

constexpr int kCellThreads = 256;
// cell index within one array: a grid's device arrays take more than 100 B a
// cell, so 2^31 cells do not fit the device
using cell_t = unsigned;

// Programmatic dependent launch: wait for the previous kernel's results, and let
// the next one's blocks be set up meanwhile (they wait in turn).  Every kernel does
// both before it touches the fields: only its own wait makes earlier launches'
// writes visible to it.  (The two launches of a CPML update do not depend on each
// other, but on what came before both; the second used to wait at its end only,
// which saved 3.6 us of a 200 x 160 x 400 step's 476.6 and rested on no promise.)
__device__ __forceinline__ void after_previous()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// the source plane at k (component-major), or null
__device__ __forceinline__ const float *src_of(const SourcePlanes &s, int k)
{
    const float *p = nullptr;
#pragma unroll
    for (int t = kMaxSourcePlanes - 1; t >= 0; t--)
        if (t < s.n && s.k[t] == k) p = s.p[t];
    return p;
}

// ---------------------------------------------------------------------------
// The Mur faces (see k_mur) of a whole step, every shell cell at once.  Face f (order x0,
// y0, z0, xE, yE, zE) sets a cell's tangential components from its old value,
// the inner neighbour's old value and the neighbour's value at that time.  A
// component is set by the faces of the two other axes only, so a cell's final
// value comes from the last of at most two faces it lies on, and where it lies
// on two, the neighbour's value at that time is what the earlier one gave it.
// Both read only cells no face sets for that component (the interior's new
// values) and the snapshot: no order between threads is needed, and the values
// are the sequential order's bit for bit.
// Needs g.old to be the snapshot of this step, taken before its E update (the
// public boundary calls may pass another: k_mur keeps the order with barriers).
// One block a plane walked its faces one after another, and the first and last
// block a whole z face: 18.9 us for the E faces of a 64^3 grid and as much for
// H's, and 24 us for the snapshot; as threads of the E and H updates, and in one
// short launch after them, they are part of the 18 us of such a step.
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T mur_scalar(const GridView<T> &g, int efield, int c, int axis, long long q, T dt, T dx)
{
    using A = Ar<T>;
    const int t = 3 - axis - c;
    const T ep = efield ? (T)g.ep[c][q] : (T)g.ep[t][q];
    const T mu = efield ? (T)g.mu[t][q] : (T)g.mu[c][q];
    const T sdt = A::mul(A::div((T)1, A::sqrt_(A::mul(ep, mu))), dt);
    return A::div(A::sub(sdt, dx), A::add(sdt, dx));
}

// The factors depend on the materials, dt and dx only, and a root and two divisions
// each are most of a shell cell's latency, up to six in a row in FP64 (the H faces'
// launch of a 64^3 grid 9.8 us, 5.9 with the factors read, its E faces in the H launch 13.9 and 9.2): a table, made when one
// of the three changes.  Per axis and face: [E or H][low or high][tangential
// component][cell of the face].
__device__ __forceinline__ long long mur_face_cell(int axis, int nx, int ny, int i, int j, int k)
{
    return axis == 0 ? j + (long long)ny * k : i + (long long)nx * (axis == 1 ? k : j);
}

__host__ __device__ __forceinline__ long long mur_face(int axis, int nx, int ny, int nz)
{
    return axis == 0 ? (long long)ny * nz : (long long)nx * (axis == 1 ? nz : ny);
}

__device__ __forceinline__ long long mur_at(int nx, int ny, int nz, int efield, int c, int axis, int hi, int i, int j, int k)
{
    const long long before = axis == 0 ? 0 : mur_face(0, nx, ny, nz) + (axis == 1 ? 0 : mur_face(1, nx, ny, nz));
    return 8 * before + (4 * (1 - efield) + 2 * hi + (c > axis ? c - 1 : c)) * mur_face(axis, nx, ny, nz) +
           mur_face_cell(axis, nx, ny, i, j, k);
}

template <typename T>
__device__ __forceinline__ T mur_factor(const GridView<T> &g, int efield, int c, int axis, int hi, int i, int j, int k)
{
    return g.mur[mur_at(g.nx, g.ny, g.nz, efield, c, axis, hi, i, j, k)];
}

template <typename T> __global__ void k_mur_table(GridView<T> g, T *out, T dt, T dx)
{
    const long long f0 = mur_face(0, g.nx, g.ny, g.nz), f1 = mur_face(1, g.nx, g.ny, g.nz), f2 = mur_face(2, g.nx, g.ny, g.nz);
    for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u < 2 * (f0 + f1 + f2);
         u += (long long)gridDim.x * blockDim.x) {
        const int hi = (int)(u & 1);
        long long t = u >> 1;
        const int axis = t < f0 ? 0 : t < f0 + f1 ? 1 : 2;
        if (axis >= 1) t -= f0;
        if (axis == 2) t -= f1;
        const int w = axis == 0 ? g.ny : g.nx, a = (int)(t % w), b = (int)(t / w);
        const int i = axis == 0 ? hi * (g.nx - 1) : a;
        const int j = axis == 0 ? a : axis == 1 ? hi * (g.ny - 1) : b;
        const int k = axis == 2 ? hi * (g.nz - 1) : b;
        const long long q = i + (long long)g.nx * (j + (long long)g.ny * k);
        for (int c = 0; c < 3; c++)
            for (int e = 0; e < 2 && c != axis; e++)
                out[mur_at(g.nx, g.ny, g.nz, e, c, axis, hi, i, j, k)] = mur_scalar(g, e, c, axis, q, dt, dx);
    }
}

template <typename T>
__device__ __forceinline__ T mur_value(T inner_old, T scalar, T inner, T own_old)
{
    using A = Ar<T>;
    return A::add(inner_old, A::mul(scalar, A::sub(inner, own_old)));
}

// cell number u of the shell: planes 0 and nz-1 whole, then the ring of the others
__device__ __forceinline__ void shell_cell(long long u, int nx, int ny, int nz, int &i, int &j, int &k)
{
    const long long nxy = (long long)nx * ny;
    if (u < 2 * nxy) {
        k = u < nxy ? 0 : nz - 1;
        const unsigned t = (unsigned)(u < nxy ? u : u - nxy);
        j = (int)(t / (unsigned)nx);
        i = (int)(t - (unsigned)j * nx);
        return;
    }
    const unsigned ring = 2u * nx + 2u * (ny - 2);
    const unsigned long long v = (unsigned long long)(u - 2 * nxy);
    const unsigned p = (unsigned)(v / ring), r = (unsigned)(v - (unsigned long long)p * ring);
    k = 1 + (int)p;
    if (r < 2u * nx) {
        j = r < (unsigned)nx ? 0 : ny - 1;
        i = (int)(r < (unsigned)nx ? r : r - nx);
    } else {
        j = 1 + (int)((r - 2u * nx) >> 1);
        i = (r & 1u) ? nx - 1 : 0;   // 2 nx is even
    }
}

// cells of the shell
__host__ __device__ __forceinline__ long long mur_cells(int nx, int ny, int nz)
{
    return 2LL * nx * ny + (nz - 2LL) * (2LL * nx + 2LL * (ny - 2));
}

// E (efield) or H of shell cell u
template <typename T>
__device__ __forceinline__ void mur_shell_cell(const GridView<T> &g, long long u, int efield)
{
    int i, j, k;
    shell_cell(u, g.nx, g.ny, g.nz, i, j, k);
    const long long nxy = (long long)g.nx * g.ny;
    const long long q = i + (long long)g.nx * j + nxy * k;
    // per axis: the face the cell lies on, in the faces' order, or -1, and the step inwards
    const int fx = i == 0 ? 0 : (i == g.nx - 1 ? 3 : -1);
    const int fy = j == 0 ? 1 : (j == g.ny - 1 ? 4 : -1);
    const int fz = k == 0 ? 2 : (k == g.nz - 1 ? 5 : -1);
    const long long dx_ = i == 0 ? 1 : -1, dy_ = j == 0 ? g.nx : -(long long)g.nx, dz_ = k == 0 ? nxy : -nxy;
    auto component = [&](int c, int a, int fa, long long da, int b, int fb, long long db) {
        if (fa < 0 && fb < 0) return;
        const bool a_last = fa > fb;
        const int last = a_last ? a : b, first = a_last ? b : a, f_last = a_last ? fa : fb, f_first = a_last ? fb : fa;
        const long long ql = q + (a_last ? da : db);
        const int m = efield ? c : 3 + c;
        const T *f = g.f[m], *old = g.old[m];
        T inner;
        if (f_first >= 0) {
            const long long qf = ql + (a_last ? db : da);
            const int in = f_last < 3 ? 1 : -1;   // ql: one step inwards along the last face's axis
            inner = mur_value(old[qf],
                              mur_factor(g, efield, c, first, f_first >= 3, i + (last == 0 ? in : 0),
                                         j + (last == 1 ? in : 0), k + (last == 2 ? in : 0)),
                              f[qf], old[ql]);
        } else {
            inner = f[ql];
        }
        g.f[m][q] = mur_value(old[ql], mur_factor(g, efield, c, last, f_last >= 3, i, j, k), inner, old[q]);
    };
    component(0, 1, fy, dy_, 2, fz, dz_);
    component(1, 0, fx, dx_, 2, fz, dz_);
    component(2, 0, fx, dx_, 1, fy, dy_);
}

// ---------------------------------------------------------------------------
// E interior.  Semi-implicit form: timefield3d_apply_E_timestep_zsection
// (timefield3d.c:1759-1837); explicit form: timefield3d_apply_E_timestep
// (timefield3d.c:1607-1677).
// ---------------------------------------------------------------------------
// update coefficients of one E component: out = main (keep e + curl - J)
template <typename T, bool SIG> __device__ __forceinline__ void e_coeffs(T ep, T sig, T dt, T &main, T &keep)
{
    using A = Ar<T>;
    const T r = A::div(ep, dt);
    if (SIG) {
        main = A::div((T)1, A::add(r, A::mul((T)0.5, sig)));
        keep = A::sub(r, A::mul((T)0.5, sig));
    } else {
        main = A::div((T)1, r);
        keep = r;
    }
}

// CPML state of one cell and field: slab-local indices, the auxiliaries of the
// slabs it lies in (else 0) and their profiles (else b = a = 0, 1/kappa = 1)
template <typename T> struct CellCpml {
    int sx, sy, sz;
    cell_t ox, oy, oz;
    T px0, px1, py0, py1, pz0, pz1;
    T bx, ax, kx, by, ay, ky, bz, az, kz;
};

// w: 0 for E, 1 for H
template <typename T>
__device__ __forceinline__ void cpml_load(CellCpml<T> &p, const CpmlView<T> &c, int nx, int ny, int nz, int i, int j,
                                          int k, cell_t ij, cell_t nxy, int w)
{
    const int L = c.L;
    p.sx = slab_local(i, nx, L);
    p.sy = slab_local(j, ny, L);
    p.sz = slab_local(k, nz, L);
    p.px0 = p.px1 = p.py0 = p.py1 = p.pz0 = p.pz1 = (T)0;
    p.bx = p.ax = p.by = p.ay = p.bz = p.az = (T)0;
    p.kx = p.ky = p.kz = (T)1;
    if (p.sx >= 0) {
        p.ox = (cell_t)p.sx + (cell_t)(2 * L) * ((cell_t)j + (cell_t)ny * (cell_t)k);
        p.px0 = c.psi[0][2 * w][p.ox];
        p.px1 = c.psi[0][2 * w + 1][p.ox];
        p.bx = c.prof[3 * w][0][i];
        p.ax = c.prof[3 * w + 1][0][i];
        p.kx = c.prof[3 * w + 2][0][i];
    }
    if (p.sy >= 0) {
        p.oy = (cell_t)i + (cell_t)nx * (cell_t)(p.sy + 2 * L * k);
        p.py0 = c.psi[1][2 * w][p.oy];
        p.py1 = c.psi[1][2 * w + 1][p.oy];
        p.by = c.prof[3 * w][1][j];
        p.ay = c.prof[3 * w + 1][1][j];
        p.ky = c.prof[3 * w + 2][1][j];
    }
    if (p.sz >= 0) {
        p.oz = ij + nxy * (cell_t)p.sz;
        p.pz0 = c.psi[2][2 * w][p.oz];
        p.pz1 = c.psi[2][2 * w + 1][p.oz];
        p.bz = c.prof[3 * w][2][k];
        p.az = c.prof[3 * w + 1][2][k];
        p.kz = c.prof[3 * w + 2][2][k];
    }
}

// the curl with its CPML terms; dU_dv: differences as the plain curl uses them
template <typename T>
__device__ __forceinline__ void cpml_curl3(CellCpml<T> &p, T divisor, T dz_dy, T dy_dz, T dx_dz, T dz_dx, T dy_dx,
                                           T dx_dy, T curl[3])
{
    using A = Ar<T>;
    if (p.sx >= 0) {
        p.px0 = A::add(A::mul(p.bx, p.px0), A::mul(p.ax, A::mul(dz_dx, divisor)));
        p.px1 = A::add(A::mul(p.bx, p.px1), A::mul(p.ax, A::mul(dy_dx, divisor)));
    }
    if (p.sy >= 0) {
        p.py0 = A::add(A::mul(p.by, p.py0), A::mul(p.ay, A::mul(dz_dy, divisor)));
        p.py1 = A::add(A::mul(p.by, p.py1), A::mul(p.ay, A::mul(dx_dy, divisor)));
    }
    if (p.sz >= 0) {
        p.pz0 = A::add(A::mul(p.bz, p.pz0), A::mul(p.az, A::mul(dy_dz, divisor)));
        p.pz1 = A::add(A::mul(p.bz, p.pz1), A::mul(p.az, A::mul(dx_dz, divisor)));
    }
    curl[0] = A::add(A::mul(divisor, A::sub(A::mul(dz_dy, p.ky), A::mul(dy_dz, p.kz))), A::sub(p.py0, p.pz0));
    curl[1] = A::add(A::mul(divisor, A::sub(A::mul(dx_dz, p.kz), A::mul(dz_dx, p.kx))), A::sub(p.pz1, p.px0));
    curl[2] = A::add(A::mul(divisor, A::sub(A::mul(dy_dx, p.kx), A::mul(dx_dy, p.ky))), A::sub(p.px1, p.py1));
}

template <typename T>
__device__ __forceinline__ void cpml_store(const CellCpml<T> &p, const CpmlView<T> &c, int w)
{
    if (p.sx >= 0) {
        c.psi[0][2 * w][p.ox] = p.px0;
        c.psi[0][2 * w + 1][p.ox] = p.px1;
    }
    if (p.sy >= 0) {
        c.psi[1][2 * w][p.oy] = p.py0;
        c.psi[1][2 * w + 1][p.oy] = p.py1;
    }
    if (p.sz >= 0) {
        c.psi[2][2 * w][p.oz] = p.pz0;
        c.psi[2][2 * w + 1][p.oz] = p.pz1;
    }
}

// The cells of a launch.  Without CPML: interior cells of planes [k_lo, k_hi)
// (every cell with a snapshot), a block's 256 consecutive in a plane.  A CPML
// grid's step takes two launches, PART 1 the cells in no slab and PART 2 those
// in one: the plain update needs 64 registers a thread and the CPML one 80 to
// 92, and at two or three blocks an SM the loads in flight do not cover their
// latency (FP64 E and H of the 200 x 160 x 400 grid: 373 and 307 us in one launch
// each, 279 and 200 in two).
// PART 0: both, for calls on a range of planes.
struct CellRange {
    int k_lo, k_hi;
    int x0, y0, w, h;      // columns and rows of a plane: [x0, x0 + w) x [y0, y0 + h)
    int L;                 // PART 2: slab thickness
};

// false: no cell of this launch
template <int PART>
__device__ __forceinline__ bool cell_of(const CellRange &r, int nx, int ny, int nz, unsigned t, int slot, int &i, int &j,
                                        int &k)
{
    if (PART != 2) {
        if (t >= (unsigned)r.w * (unsigned)r.h) return false;
        const int y = (int)(t / (unsigned)r.w);
        i = r.x0 + (int)(t - (unsigned)y * (unsigned)r.w);
        j = r.y0 + y;
        k = r.k_lo + slot;
        return true;
    }
    // cells in one row: the 2L - 2 updated planes of the z slabs, whole, then of
    // each middle plane the 2L - 2 rows of the y slabs and, in the other rows, the
    // 2L - 2 columns of the x slabs
    const unsigned S = (unsigned)r.L - 1, W = (unsigned)nx - 2, H = (unsigned)ny - 2, mid = (unsigned)(ny - 2 * r.L);
    const unsigned plane = W * H, zcells = 2 * S * plane;
    if (t < zcells) {
        const unsigned z = t / plane;
        t -= z * plane;
        const unsigned y = t / W;
        k = (int)(z < S ? 1 + z : (unsigned)(nz - r.L) + z - S);
        j = 1 + (int)y;
        i = 1 + (int)(t - y * W);
        return true;
    }
    t -= zcells;
    const unsigned rows = 2 * S * W, ring = rows + 2 * S * mid;
    const unsigned z = t / ring;
    if (z >= (unsigned)(nz - 2 * r.L)) return false;
    t -= z * ring;
    k = r.L + (int)z;
    if (t < rows) {
        const unsigned y = t / W;
        j = (int)(y < S ? 1 + y : (unsigned)(ny - r.L) + y - S);
        i = 1 + (int)(t - y * W);
        return true;
    }
    t -= rows;
    const unsigned y = t / (2 * S), x = t - y * (2 * S);
    j = r.L + (int)y;
    i = (int)(x < S ? 1 + x : (unsigned)(nx - r.L) + x - S);
    return true;
}

// slots (planes) and cells of a slot of a launch
static void cell_extent(const CellRange &r, int nx, int ny, int nz, int part, int &slots, long long &cells)
{
    if (part != 2) {
        slots = r.k_hi - r.k_lo;
        cells = (long long)r.w * r.h;
        return;
    }
    const long long S = r.L - 1, W = nx - 2, H = ny - 2;
    slots = 1;
    cells = 2 * S * W * H + (nz - 2LL * r.L) * (2 * S * W + 2 * S * (ny - 2LL * r.L));
}

// SNAP: the launch covers every cell and first copies the 2-cell shell of all
// six components to g.old (timefield3d_update_old_edge_fields,
// timefield3d.c:246-346): the Mur step's snapshot, taken while the cell is in
// registers instead of in a launch of its own
template <typename T, bool SIG, bool CPML, bool EXPL, bool SNAP, int PART>
__global__ void __launch_bounds__(kCellThreads, CPML ? 3 : 4)
k_update_E(GridView<T> g, CpmlView<T> c, SourcePlanes src, T dt, T divisor, CellRange r, int slots)
{
    using A = Ar<T>;
    after_previous();
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const cell_t nxy = (cell_t)nx * (cell_t)ny;
    for (int slot = blockIdx.y; slot < slots; slot += gridDim.y) {
        int i, j, k;
        if (!cell_of<PART>(r, nx, ny, nz, blockIdx.x * (unsigned)kCellThreads + threadIdx.x, slot, i, j, k)) continue;
        const cell_t ij = (cell_t)i + (cell_t)nx * (cell_t)j, q = ij + nxy * (cell_t)k;
        T e[3];
        if (SNAP) {
            const bool shell = i <= 1 || i >= nx - 2 || j <= 1 || j >= ny - 2 || k <= 1 || k >= nz - 2;
            if (shell) {
#pragma unroll
                for (int m = 0; m < 6; m++) g.old[m][q] = g.f[m][q];
            }
            if (i < 1 || i > nx - 2 || j < 1 || j > ny - 2 || k < 1 || k > nz - 2) continue;
        }
        const float *sp = src_of(src, k);
        const T hx = g.f[3][q], hy = g.f[4][q], hz = g.f[5][q];
        const T hx_j = g.f[3][q - nx], hz_j = g.f[5][q - nx];
        const T hx_k = g.f[3][q - nxy], hy_k = g.f[4][q - nxy];
        const T hy_i = g.f[4][q - 1], hz_i = g.f[5][q - 1];
        T ep[3], sig[3];
#pragma unroll
        for (int m = 0; m < 3; m++) {
            e[m] = g.f[m][q];
            ep[m] = (T)g.ep[m][q];
            sig[m] = SIG ? (T)g.sig[m][q] : (T)0;
        }
        CellCpml<T> p;
        if (CPML) cpml_load(p, c, nx, ny, nz, i, j, k, ij, nxy, 0);
        const T dHz_dy = A::sub(hz, hz_j), dHy_dz = A::sub(hy, hy_k), dHx_dz = A::sub(hx, hx_k);
        const T dHz_dx = A::sub(hz, hz_i), dHy_dx = A::sub(hy, hy_i), dHx_dy = A::sub(hx, hx_j);
        T curl[3];
        if (CPML) {
            cpml_curl3(p, divisor, dHz_dy, dHy_dz, dHx_dz, dHz_dx, dHy_dx, dHx_dy, curl);
        } else {
            curl[0] = A::mul(divisor, A::sub(dHz_dy, dHy_dz));
            curl[1] = A::mul(divisor, A::sub(dHx_dz, dHz_dx));
            curl[2] = A::mul(divisor, A::sub(dHy_dx, dHx_dy));
        }
        T main = 0, keep = 0;
#pragma unroll
        for (int m = 0; m < 3; m++) {
            const T J = sp ? (T)sp[m * nxy + ij] : (T)0;
            if (EXPL) {
                const T Jt = A::add(J, A::mul(e[m], sig[m]));
                e[m] = A::add(e[m], A::div(A::mul(dt, A::sub(curl[m], Jt)), ep[m]));
            } else {
                if (m == 0 || ep[m] != ep[m - 1] || (SIG && sig[m] != sig[m - 1]))
                    e_coeffs<T, SIG>(ep[m], sig[m], dt, main, keep);
                e[m] = A::mul(main, A::sub(A::add(A::mul(keep, e[m]), curl[m]), J));
            }
        }
#pragma unroll
        for (int m = 0; m < 3; m++) g.f[m][q] = e[m];
        if (CPML) cpml_store(p, c, 0);
    }
}

// ---------------------------------------------------------------------------
// H interior.  Semi-implicit: timefield3d_apply_H_timestep_zsection
// (timefield3d.c:1679-1757), magnetic current = source + sig_m H
// (timefield3d.c:1705-1707); explicit: timefield3d_apply_H_timestep
// (timefield3d.c:1537-1605).
// ---------------------------------------------------------------------------
// h_coeff, h_main: 1/dt and 1/(1/dt), the coefficients where mu = 1 and no loss
// MUR: the launch also sets E on the shell (the E faces of the Mur step): slots
// before the planes are the shell's cells.  An interior cell whose +x, +y or +z
// neighbour is on the shell needs that face's new E and computes it itself --
// such a neighbour lies on one face only, and its inner neighbour is the cell --
// so H waits for no launch of its own between the two.
template <typename T, bool SIG, bool MU, bool CPML, bool EXPL, int PART, bool MUR>
__global__ void __launch_bounds__(kCellThreads, CPML ? 3 : 4)
k_update_H(GridView<T> g, CpmlView<T> c, SourcePlanes src, T dt, T divisor, T h_coeff, T h_main, CellRange r, int slots)
{
    using A = Ar<T>;
    after_previous();
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const cell_t nxy = (cell_t)nx * (cell_t)ny;
    const int shell_slots = MUR ? (int)((mur_cells(nx, ny, nz) + gridDim.x * kCellThreads - 1) /
                                        (gridDim.x * kCellThreads)) : 0;
    for (int slot = (int)blockIdx.y - shell_slots; slot < slots; slot += gridDim.y) {
        int i, j, k;
        if (MUR && slot < 0) {   // the shell first: its cells take the longest
            const long long u = ((long long)(slot + shell_slots) * gridDim.x + blockIdx.x) * kCellThreads + threadIdx.x;
            if (u < mur_cells(nx, ny, nz)) mur_shell_cell(g, u, 1);
            continue;
        }
        // backwards: H starts on what E left in L2, and E on what H did
        const unsigned bx = PART == 2 ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
        if (!cell_of<PART>(r, nx, ny, nz, bx * (unsigned)kCellThreads + threadIdx.x, slots - 1 - slot, i, j, k)) continue;
        const cell_t ij = (cell_t)i + (cell_t)nx * (cell_t)j, q = ij + nxy * (cell_t)k;
        const float *sp = src_of(src, k);
        const T ex = g.f[0][q], ey = g.f[1][q], ez = g.f[2][q];
        T ex_j, ez_j, ex_k, ey_k, ey_i, ez_i;
        auto next = [&](int c, T inner, int axis, cell_t qn, bool face) -> T {
            return MUR && face ? mur_value(g.old[c][q], mur_factor(g, 1, c, axis, 1, i, j, k), inner, g.old[c][qn])
                               : g.f[c][qn];
        };
        ex_j = next(0, ex, 1, q + nx, j == ny - 2);
        ez_j = next(2, ez, 1, q + nx, j == ny - 2);
        ex_k = next(0, ex, 2, q + nxy, k == nz - 2);
        ey_k = next(1, ey, 2, q + nxy, k == nz - 2);
        ey_i = next(1, ey, 0, q + 1, i == nx - 2);
        ez_i = next(2, ez, 0, q + 1, i == nx - 2);
        T h[3], mu[3], sig[3];
#pragma unroll
        for (int m = 0; m < 3; m++) {
            h[m] = g.f[3 + m][q];
            mu[m] = MU ? (T)g.mu[m][q] : (T)1;
            sig[m] = SIG ? (T)g.sig[3 + m][q] : (T)0;
        }
        CellCpml<T> p;
        if (CPML) cpml_load(p, c, nx, ny, nz, i, j, k, ij, nxy, 1);
        const T dEz_dy = A::sub(ez_j, ez), dEy_dz = A::sub(ey_k, ey), dEx_dz = A::sub(ex_k, ex);
        const T dEz_dx = A::sub(ez_i, ez), dEy_dx = A::sub(ey_i, ey), dEx_dy = A::sub(ex_j, ex);
        T curl[3];
        if (CPML) {
            cpml_curl3(p, divisor, dEz_dy, dEy_dz, dEx_dz, dEz_dx, dEy_dx, dEx_dy, curl);
        } else {
            curl[0] = A::mul(divisor, A::sub(dEz_dy, dEy_dz));
            curl[1] = A::mul(divisor, A::sub(dEx_dz, dEz_dx));
            curl[2] = A::mul(divisor, A::sub(dEy_dx, dEx_dy));
        }
        T main = h_main, keep = h_coeff;
#pragma unroll
        for (int m = 0; m < 3; m++) {
            T M = sp ? (T)sp[(3 + m) * nxy + ij] : (T)0;
            if (SIG) M = A::add(M, A::mul(h[m], sig[m]));
            if (EXPL) {
                h[m] = A::sub(h[m], A::div(A::mul(dt, A::add(curl[m], M)), mu[m]));
            } else {
                if ((SIG || MU) && (m == 0 || mu[m] != mu[m - 1] || (SIG && sig[m] != sig[m - 1])))
                    e_coeffs<T, SIG>(mu[m], sig[m], dt, main, keep);
                h[m] = A::mul(main, A::sub(A::sub(A::mul(keep, h[m]), curl[m]), M));
            }
        }
#pragma unroll
        for (int m = 0; m < 3; m++) g.f[3 + m][q] = h[m];
        if (CPML) cpml_store(p, c, 1);
    }
}

// ---------------------------------------------------------------------------
// Shell snapshot: timefield3d_update_old_edge_fields (timefield3d.c:246-346),
// the 2-cell shell of all six components.  One block per z plane: planes
// 0,1,nz-2,nz-1 entirely, other planes only their 2-cell ring.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void k_save_shell(GridView<T> g)
{
    const int k = blockIdx.x;
    const long long nxy = (long long)g.nx * g.ny;
    const long long base = nxy * k;
    const bool full = k <= 1 || k >= g.nz - 2;
    if (full) {
        for (long long t = threadIdx.x; t < nxy; t += blockDim.x)
#pragma unroll
            for (int m = 0; m < 6; m++) g.old[m][base + t] = g.f[m][base + t];
        return;
    }
    // ring: rows 0,1,ny-2,ny-1 whole; other rows columns 0,1,nx-2,nx-1
    const int nrow_full = 4 * g.nx;
    const int nring = nrow_full + 4 * (g.ny - 4);
    for (int t = threadIdx.x; t < nring; t += blockDim.x) {
        int i, j;
        if (t < nrow_full) {
            int r = t / g.nx;
            i = t - r * g.nx;
            j = r < 2 ? r : g.ny - 4 + r;
        } else {
            int u = t - nrow_full;
            int r = u >> 2, cidx = u & 3;
            j = 2 + r;
            i = cidx < 2 ? cidx : g.nx - 4 + cidx;
        }
        long long q = base + i + (long long)g.nx * j;
#pragma unroll
        for (int m = 0; m < 6; m++) g.old[m][q] = g.f[m][q];
    }
}

// ---------------------------------------------------------------------------
// Mur first-order ABC, E (timefield3d.c:2499-2721) or H (2275-2497) faces.
// Faces run in the reference's order x=0, y=0, z=0, x=end, y=end, z=end and
// later faces read what earlier ones wrote on shared edges, so the order is
// kept inside a block.  x and y faces only couple cells of one z plane, so a
// block owns one plane; the first block also owns plane 1 and runs the z=0
// face after that plane's x=0/y=0 faces (its inner cells), the last block
// likewise for the z=end face.  Tangential components of a face normal to a:
// x: (y,z), y: (x,z), z: (x,y); for E component c v = 1/sqrt(ep_c mu_t), for
// H component c v = 1/sqrt(ep_t mu_c), t the third axis.
// ---------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void mur_cell(GridView<T> &g, int efield, int axis, long long qb, long long qi,
                                          T dt, T dx)
{
    using A = Ar<T>;
    const int c1 = axis == 0 ? 1 : 0, c2 = axis == 2 ? 1 : 2;
#pragma unroll
    for (int w = 0; w < 2; w++) {
        int c = w ? c2 : c1;
        int t = 3 - axis - c;
        T ep = efield ? (T)g.ep[c][qb] : (T)g.ep[t][qb];
        T mu = efield ? (T)g.mu[t][qb] : (T)g.mu[c][qb];
        int m = efield ? c : 3 + c;
        T F_old = g.old[m][qb];
        T F_inner = g.f[m][qi];
        T F_inner_old = g.old[m][qi];
        T speed = A::div((T)1, A::sqrt_(A::mul(ep, mu)));
        T sdt = A::mul(speed, dt);
        T scalar = A::div(A::sub(sdt, dx), A::add(sdt, dx));
        g.f[m][qb] = A::add(F_inner_old, A::mul(scalar, A::sub(F_inner, F_old)));
    }
}

template <typename T>
__global__ void k_mur(GridView<T> g, T dt, T dx, int efield, int ks, int ke)
{
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const long long nxy = (long long)nx * ny;
    const int lo = ks == 0, hi = ke == nz;
    const int mid0 = lo ? 2 : ks, mid1 = hi ? nz - 2 : ke;
    const int nblk = lo + max(0, mid1 - mid0) + hi;
    const int b = blockIdx.x;
    if (b >= nblk) return;
    int p0, p1, zface = -1;
    if (lo && b == 0) { p0 = 0; p1 = min(2, ke); zface = 0; }
    else if (hi && b == nblk - 1) { p0 = nz - 2; p1 = nz; zface = 1; }
    else { p0 = mid0 + b - lo; p1 = p0 + 1; }
    const int np = p1 - p0;
    for (int high = 0; high < 2; high++) {
        // x face
        {
            int ib = high ? nx - 1 : 0, ii = high ? nx - 2 : 1;
            for (int t = threadIdx.x; t < ny * np; t += blockDim.x) {
                int j = t % ny, k = p0 + t / ny;
                long long r = (long long)nx * j + nxy * k;
                mur_cell(g, efield, 0, r + ib, r + ii, dt, dx);
            }
        }
        __syncthreads();
        // y face
        {
            int jb = high ? ny - 1 : 0, ji = high ? ny - 2 : 1;
            for (int t = threadIdx.x; t < nx * np; t += blockDim.x) {
                int i = t % nx, k = p0 + t / nx;
                long long r = i + nxy * k;
                mur_cell(g, efield, 1, r + (long long)nx * jb, r + (long long)nx * ji, dt, dx);
            }
        }
        __syncthreads();
        // z face
        if (zface == high) {
            int kb = high ? nz - 1 : 0, ki = high ? nz - 2 : 1;
            for (long long t = threadIdx.x; t < nxy; t += blockDim.x)
                mur_cell(g, efield, 2, t + nxy * kb, t + nxy * ki, dt, dx);
        }
        __syncthreads();
    }
}

// H faces of a step, the probes (interior ones: no face sets them) and the step
// counter
template <typename T>
__global__ void __launch_bounds__(kCellThreads) k_mur_step(GridView<T> g, StepEnd end)
{
    after_previous();
    if (blockIdx.x == gridDim.x - 1) {
        for (int p = threadIdx.x; p < end.np; p += kCellThreads) {
            const int n = end.count[p];
            if (n < end.cap) end.buf[(long long)p * end.cap + n] = (double)g.f[end.probes[p].m][end.probes[p].q];
            end.count[p] = n + 1;
        }
        if (threadIdx.x == 0 && end.step) *end.step += 1;
        return;
    }
    const long long u = blockIdx.x * (long long)kCellThreads + threadIdx.x;
    if (u < mur_cells(g.nx, g.ny, g.nz)) mur_shell_cell(g, u, 0);
}

// AoS double (reference layout) -> SoA T, whole grid
template <typename T>
__global__ void k_aos_to_soa(const double *aos, T *d0, T *d1, T *d2, T *d3, T *d4, T *d5, long long n)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const double *a = aos + 6 * q;
        d0[q] = (T)a[0]; d1[q] = (T)a[1]; d2[q] = (T)a[2];
        d3[q] = (T)a[3]; d4[q] = (T)a[4]; d5[q] = (T)a[5];
    }
}

// SoA T -> AoS double
template <typename T>
__global__ void k_soa_to_aos(double *aos, const T *s0, const T *s1, const T *s2, const T *s3, const T *s4,
                             const T *s5, long long n)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        double *a = aos + 6 * q;
        a[0] = (double)s0[q]; a[1] = (double)s1[q]; a[2] = (double)s2[q];
        a[3] = (double)s3[q]; a[4] = (double)s4[q]; a[5] = (double)s5[q];
    }
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
// launch with a programmatic dependency on the preceding kernel (after_previous)
template <typename... P, typename... A>
static void launch_cells(void (*k)(P...), dim3 grid, cudaStream_t st, A... args)
{
    note_launch();
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kCellThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k, P(args)...);
}

template <typename F> static void for_range(const CellRange &r, int nx, int ny, int nz, int part, F f)
{
    int slots;
    long long cells;
    cell_extent(r, nx, ny, nz, part, slots, cells);
    if (slots <= 0 || cells <= 0) return;
    f(dim3((unsigned)((cells + kCellThreads - 1) / kCellThreads), (unsigned)(slots < 65535 ? slots : 65535)), slots);
}

// interior cells of planes [k_lo, k_hi), or (snapshot) every cell
static CellRange cell_range(int nx, int ny, int nz, int k_lo, int k_hi, bool snapshot)
{
    if (snapshot) return CellRange{0, nz, 0, 0, nx, ny, 0};
    return CellRange{k_lo < 1 ? 1 : k_lo, k_hi > nz - 1 ? nz - 1 : k_hi, 1, 1, nx - 2, ny - 2, 0};
}

// the cells of a CPML grid in no slab
static CellRange slab_free(int nx, int ny, int nz, int L)
{
    return CellRange{L, nz - L, L, L, nx - 2 * L, ny - 2 * L, L};
}

template <typename T>
void launch_update_E(const GridView<T> &g, const CpmlView<T> &c, const SourcePlanes &s, T dt, T divisor,
                     int k_lo, int k_hi, bool sig, bool cpml, bool expl, bool snapshot, cudaStream_t st)
{
    const CellRange all = cell_range(g.nx, g.ny, g.nz, k_lo, k_hi, snapshot);
    const bool whole = cpml && c.L >= 1 && all.k_lo == 1 && all.k_hi == g.nz - 1;
#define FDTD_E(RANGE, ...)                                                                            \
    for_range(RANGE, g.nx, g.ny, g.nz, part, [&](dim3 grd, int slots) {                               \
        launch_cells(k_update_E<T, __VA_ARGS__>, grd, st, g, c, s, dt, divisor, RANGE, slots);        \
    })
    int part = 0;
    if (expl) FDTD_E(all, true, false, true, false, 0);
    else if (whole) {
        const CellRange in = slab_free(g.nx, g.ny, g.nz, c.L);
        part = 1;
        if (sig) FDTD_E(in, true, false, false, false, 1); else FDTD_E(in, false, false, false, false, 1);
        part = 2;
        if (sig) FDTD_E(in, true, true, false, false, 2); else FDTD_E(in, false, true, false, false, 2);
    }
    else if (cpml) { if (sig) FDTD_E(all, true, true, false, false, 0); else FDTD_E(all, false, true, false, false, 0); }
    else if (snapshot) { if (sig) FDTD_E(all, true, false, false, true, 0); else FDTD_E(all, false, false, false, true, 0); }
    else { if (sig) FDTD_E(all, true, false, false, false, 0); else FDTD_E(all, false, false, false, false, 0); }
#undef FDTD_E
}

template <typename T>
void launch_update_H(const GridView<T> &g, const CpmlView<T> &c, const SourcePlanes &s, T dt, T divisor,
                     int k_lo, int k_hi, bool sig, bool mu, bool cpml, bool expl, bool faces, cudaStream_t st)
{
    const CellRange all = cell_range(g.nx, g.ny, g.nz, k_lo, k_hi, false);
    const T h_coeff = (T)1 / dt, h_main = (T)1 / h_coeff;
    const bool whole = cpml && c.L >= 1 && all.k_lo == 1 && all.k_hi == g.nz - 1;
#define FDTD_H(RANGE, ...)                                                                                          \
    for_range(RANGE, g.nx, g.ny, g.nz, part, [&](dim3 grd, int slots) {                                             \
        if (faces) grd.y = (unsigned)std::min<long long>(65535, grd.y + mur_cells(g.nx, g.ny, g.nz) / ((long long)grd.x * kCellThreads) + 1); \
        launch_cells(k_update_H<T, __VA_ARGS__>, grd, st, g, c, s, dt, divisor, h_coeff, h_main, RANGE, slots); \
    })
#define FDTD_H3(RANGE, CP, PT, FACES)                                     \
    do {                                                                  \
        if (sig) FDTD_H(RANGE, true, true, CP, false, PT, FACES);         \
        else if (mu) FDTD_H(RANGE, false, true, CP, false, PT, FACES);    \
        else FDTD_H(RANGE, false, false, CP, false, PT, FACES);           \
    } while (0)
    int part = 0;
    if (expl) FDTD_H(all, true, true, false, true, 0, false);
    else if (whole) {
        const CellRange in = slab_free(g.nx, g.ny, g.nz, c.L);
        part = 1;
        FDTD_H3(in, false, 1, false);
        part = 2;
        FDTD_H3(in, true, 2, false);
    }
    else if (cpml) FDTD_H3(all, true, 0, false);
    else if (faces) FDTD_H3(all, false, 0, true);
    else FDTD_H3(all, false, 0, false);
#undef FDTD_H3
#undef FDTD_H
}

template <typename T> void launch_mur_step(const GridView<T> &g, const StepEnd &end, cudaStream_t st)
{
    const long long blocks = (mur_cells(g.nx, g.ny, g.nz) + kCellThreads - 1) / kCellThreads + 1;
    launch_cells(k_mur_step<T>, dim3((unsigned)blocks), st, g, end);
}

long long mur_table_size(int nx, int ny, int nz)
{
    return 8 * (mur_face(0, nx, ny, nz) + mur_face(1, nx, ny, nz) + mur_face(2, nx, ny, nz));
}

template <typename T> void launch_mur_table(const GridView<T> &g, T *out, T dt, T dx, cudaStream_t st)
{
    note_launch();
    const long long blocks = (mur_table_size(g.nx, g.ny, g.nz) / 4 + 255) / 256;
    k_mur_table<T><<<(unsigned)std::min<long long>(blocks, 4736), 256, 0, st>>>(g, out, dt, dx);
}

template <typename T>
void launch_save_shell(const GridView<T> &g, cudaStream_t st)
{
    note_launch();
    k_save_shell<T><<<g.nz, 256, 0, st>>>(g);
}

template <typename T>
void launch_mur(const GridView<T> &g, T dt, T dx, int efield, int ks, int ke, cudaStream_t st)
{
    const int lo = ks == 0, hi = ke == g.nz;
    const int mid0 = lo ? 2 : ks, mid1 = hi ? g.nz - 2 : ke;
    int nblk = lo + (mid1 > mid0 ? mid1 - mid0 : 0) + hi;
    if (nblk > 0) {
        note_launch();
        k_mur<T><<<nblk, 256, 0, st>>>(g, dt, dx, efield, ks, ke);
    }
}

template <typename T>
void launch_aos_to_soa(const double *aos, T *const d[6], long long n, cudaStream_t st)
{
    int blocks = (int)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096);
    note_launch();
    k_aos_to_soa<T><<<blocks, 256, 0, st>>>(aos, d[0], d[1], d[2], d[3], d[4], d[5], n);
}

template <typename T>
void launch_soa_to_aos(double *aos, T *const s[6], long long n, cudaStream_t st)
{
    int blocks = (int)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096);
    note_launch();
    k_soa_to_aos<T><<<blocks, 256, 0, st>>>(aos, s[0], s[1], s[2], s[3], s[4], s[5], n);
}

#define FDTD_INST(T)                                                                                          \
    template void launch_update_E<T>(const GridView<T> &, const CpmlView<T> &, const SourcePlanes &, T, T, int, \
                                     int, bool, bool, bool, bool, cudaStream_t);                               \
    template void launch_mur_step<T>(const GridView<T> &, const StepEnd &, cudaStream_t);                     \
    template void launch_mur_table<T>(const GridView<T> &, T *, T, T, cudaStream_t);                          \
    template void launch_update_H<T>(const GridView<T> &, const CpmlView<T> &, const SourcePlanes &, T, T, int, \
                                     int, bool, bool, bool, bool, bool, cudaStream_t);                         \
    template void launch_save_shell<T>(const GridView<T> &, cudaStream_t);                                    \
    template void launch_mur<T>(const GridView<T> &, T, T, int, int, int, cudaStream_t);                       \
    template void launch_aos_to_soa<T>(const double *, T *const[6], long long, cudaStream_t);                  \
    template void launch_soa_to_aos<T>(double *, T *const[6], long long, cudaStream_t);
FDTD_INST(float)
FDTD_INST(double)
#undef FDTD_INST

}  // namespace fdtd
