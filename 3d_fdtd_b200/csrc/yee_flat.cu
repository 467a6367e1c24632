// yee_flat.cu -- FP32 Yee step as two flat kernels, a thread a cell: E from H, then
// H from the new E, both in place.  For grids that no streaming kernel takes (rows
// that are no multiple of four cells) and on request.
//
// Bound by memory: E reads E, H and its coefficients and writes E (48 B a cell, 40
// where the three coefficients are one array), H reads both and writes H (36 B), and
// a slab cell moves 16 B more in each for every slab it lies in.  Neighbours come
// from L1 and L2.  A block is 256 consecutive cells of a plane and issues every load
// of a cell before its arithmetic and stores.  The slabs' cells are blocks of their
// own, first in the launch: interior cells carry no slab test, and a thread takes
// three planes of them, which shares the index arithmetic and the z neighbours (with
// the slabs' registers it costs occupancy: 107 us).  H takes the blocks backwards, so
// that each kernel starts on what the other left in L2.  157x131x203 cells with a
// 10-cell CPML, us a step: 152 as tiles of 32 x 8 cells with slab tests and loads
// behind one another in 64-bit indices; 90 with the loads first and slabs apart; 84
// with H backwards; 72.5, 68 and 72 with two, three and four planes a thread.  (76 B a
// cell and the slabs' are 55 us at the rate of a copy.)  199x161x399: 481, now 222.
//
// Arithmetic is the fused kernels' (FP32, raw curl differences):
//   E' = ca E + cb (curl_H + dx (psi_a - psi_b) - dx J)
//   H' = H - hb (curl_E + dx (psi_a - psi_b) + dx M),   hb = dt/dx
// with psi' = b psi + a (difference / dx) inside the CPML slabs, the units of the
// split FP64 kernels and the CPU restatement.
#include "common.cuh"
#include "kernels.h"

#include <algorithm>

namespace fdtd {

constexpr int kFlatThreads = 256;
// cell index within one array: a grid's device arrays take more than 60 B a cell,
// so 2^32 cells do not fit the device
using cell_t = unsigned;

// `w` columns of the rows [j0, j0 + rows) of planes [k0, k1), in blocks of 256 cells,
// `per` a plane (of the box, a thread's kFlatZ planes).  The cells in z slabs, the
// others in y slabs, the others in x slabs (columns left and right), then the box.
constexpr int kFlatZ = 3, kFlatX = 4, kFlatBox = 5, kFlatRegions = 6;
struct FlatRegion {
    unsigned first, per;
    int w, j0, rows, k0, k1;
};
struct FlatRange {
    FlatRegion r[kFlatRegions];
};

__device__ __forceinline__ const float *flat_src(const SourcePlanes &s, int k)
{
    const float *p = nullptr;
#pragma unroll
    for (int t = kMaxSourcePlanes - 1; t >= 0; t--)
        if (t < s.n && s.k[t] == k) p = s.p[t];
    return p;
}

// the auxiliaries of a slab cell (W 0: of E, 1: of H), and its curl
struct FlatPsi {
    int sx, sy, sz;
    cell_t ox, oy, oz;
    float x0, x1, y0, y1, z0, z1;
};

template <int W>
__device__ __forceinline__ void flat_psi_load(FlatPsi &p, const FlatArgs &a, int i, int j, int k, cell_t ij, cell_t nxy)
{
    const int L = a.L;
    p.sx = slab_local(i, a.nx, L);
    p.sy = slab_local(j, a.ny, L);
    p.sz = slab_local(k, a.nz, L);
    p.x0 = p.x1 = p.y0 = p.y1 = p.z0 = p.z1 = 0.f;
    p.ox = p.oy = p.oz = 0;
    if (p.sx >= 0) {
        p.ox = (cell_t)p.sx + (cell_t)(2 * L) * ((cell_t)j + (cell_t)a.ny * (cell_t)k);
        p.x0 = a.psi[0][2 * W][p.ox];
        p.x1 = a.psi[0][2 * W + 1][p.ox];
    }
    if (p.sy >= 0) {
        p.oy = (cell_t)i + (cell_t)a.nx * (cell_t)(p.sy + 2 * L * k);
        p.y0 = a.psi[1][2 * W][p.oy];
        p.y1 = a.psi[1][2 * W + 1][p.oy];
    }
    if (p.sz >= 0) {
        p.oz = ij + nxy * (cell_t)p.sz;
        p.z0 = a.psi[2][2 * W][p.oz];
        p.z1 = a.psi[2][2 * W + 1][p.oz];
    }
}

template <int W>
__device__ __forceinline__ void flat_psi_curl(FlatPsi &p, const FlatArgs &a, int i, int j, int k, float dz_dy,
                                              float dy_dz, float dx_dz, float dz_dx, float dy_dx, float dx_dy, float c[3])
{
    const float dx = a.dx, div = 1.0f / dx;
    float kx = 1.f, ky = 1.f, kz = 1.f;
    if (p.sx >= 0) {
        const float b = __ldg(a.prof[3 * W][0] + i), s = __ldg(a.prof[3 * W + 1][0] + i);
        kx = __ldg(a.prof[3 * W + 2][0] + i);
        p.x0 = b * p.x0 + s * (dz_dx * div);
        p.x1 = b * p.x1 + s * (dy_dx * div);
        a.psi[0][2 * W][p.ox] = p.x0;
        a.psi[0][2 * W + 1][p.ox] = p.x1;
    }
    if (p.sy >= 0) {
        const float b = __ldg(a.prof[3 * W][1] + j), s = __ldg(a.prof[3 * W + 1][1] + j);
        ky = __ldg(a.prof[3 * W + 2][1] + j);
        p.y0 = b * p.y0 + s * (dz_dy * div);
        p.y1 = b * p.y1 + s * (dx_dy * div);
        a.psi[1][2 * W][p.oy] = p.y0;
        a.psi[1][2 * W + 1][p.oy] = p.y1;
    }
    if (p.sz >= 0) {
        const float b = __ldg(a.prof[3 * W][2] + k), s = __ldg(a.prof[3 * W + 1][2] + k);
        kz = __ldg(a.prof[3 * W + 2][2] + k);
        p.z0 = b * p.z0 + s * (dy_dz * div);
        p.z1 = b * p.z1 + s * (dx_dz * div);
        a.psi[2][2 * W][p.oz] = p.z0;
        a.psi[2][2 * W + 1][p.oz] = p.z1;
    }
    c[0] = ky * dz_dy - kz * dy_dz + dx * (p.y0 - p.z0);
    c[1] = kz * dx_dz - kx * dz_dx + dx * (p.z1 - p.x0);
    c[2] = kx * dy_dx - ky * dx_dy + dx * (p.x1 - p.y1);
}

// E of cell (i, j) of planes k .. k + Z - 1 (below k1)
template <int Z, bool SLAB, bool LOSSY, bool ONE>
__device__ __forceinline__ void flat_E_cells(const FlatArgs &a, int i, int j, int k, int k1)
{
    const int nx = a.nx;
    const cell_t nxy = (cell_t)nx * (cell_t)a.ny, ij = (cell_t)i + (cell_t)nx * (cell_t)j;
    const float *Hx = a.f[3], *Hy = a.f[4], *Hz = a.f[5];   // the kernel before wrote them: no __ldg
    float hx[Z + 1], hy[Z + 1], hz[Z], hx_j[Z], hz_j[Z], hy_i[Z], hz_i[Z];
    float e[Z][3], b[Z][3], keep[Z][3];
    FlatPsi p[Z];
    const cell_t q0 = ij + nxy * (cell_t)k;
    hx[0] = Hx[q0 - nxy];
    hy[0] = Hy[q0 - nxy];
#pragma unroll
    for (int z = 0; z < Z; z++) {
        const int kz = k + z < k1 ? k + z : k;   // (a plane past the end repeats the first, and is not stored)
        const cell_t q = ij + nxy * (cell_t)kz;
        hx[z + 1] = Hx[q];
        hy[z + 1] = Hy[q];
        hz[z] = Hz[q];
        hx_j[z] = Hx[q - nx];
        hz_j[z] = Hz[q - nx];
        hy_i[z] = Hy[q - 1];
        hz_i[z] = Hz[q - 1];
#pragma unroll
        for (int m = 0; m < 3; m++) {
            e[z][m] = a.f[m][q];
            b[z][m] = m == 0 || !ONE ? __ldg(a.cb[m] + q) : b[z][0];
            if (LOSSY) keep[z][m] = m == 0 || !ONE ? __ldg(a.ca[m] + q) : keep[z][0];
        }
        if (SLAB) flat_psi_load<0>(p[z], a, i, j, kz, ij, nxy);
    }
#pragma unroll
    for (int z = 0; z < Z; z++) {
        if (k + z >= k1) break;
        const cell_t q = q0 + nxy * (cell_t)z;
        const float dHz_dy = hz[z] - hz_j[z], dHy_dz = hy[z + 1] - hy[z], dHx_dz = hx[z + 1] - hx[z];
        const float dHz_dx = hz[z] - hz_i[z], dHy_dx = hy[z + 1] - hy_i[z], dHx_dy = hx[z + 1] - hx_j[z];
        float c[3];
        if (SLAB) {
            flat_psi_curl<0>(p[z], a, i, j, k + z, dHz_dy, dHy_dz, dHx_dz, dHz_dx, dHy_dx, dHx_dy, c);
        } else {
            c[0] = dHz_dy - dHy_dz;
            c[1] = dHx_dz - dHz_dx;
            c[2] = dHy_dx - dHx_dy;
        }
        if (a.src.n) {
            const float *sp = flat_src(a.src, k + z);
            if (sp) {
#pragma unroll
                for (int m = 0; m < 3; m++) c[m] -= a.dx * sp[(cell_t)m * nxy + ij];
            }
        }
#pragma unroll
        for (int m = 0; m < 3; m++) a.f[m][q] = (LOSSY ? keep[z][m] * e[z][m] : e[z][m]) + b[z][m] * c[m];
    }
}

template <int Z, bool SLAB>
__device__ __forceinline__ void flat_H_cells(const FlatArgs &a, int i, int j, int k, int k1)
{
    const int nx = a.nx;
    const cell_t nxy = (cell_t)nx * (cell_t)a.ny, ij = (cell_t)i + (cell_t)nx * (cell_t)j;
    const float *Ex = a.f[0], *Ey = a.f[1], *Ez = a.f[2];
    float ex[Z + 1], ey[Z + 1], ez[Z], ex_j[Z], ez_j[Z], ey_i[Z], ez_i[Z];
    float h[Z][3];
    FlatPsi p[Z];
    const cell_t q0 = ij + nxy * (cell_t)k;
    ex[0] = Ex[q0];
    ey[0] = Ey[q0];
#pragma unroll
    for (int z = 0; z < Z; z++) {
        const int kz = k + z < k1 ? k + z : k;
        const cell_t q = ij + nxy * (cell_t)kz;
        ex[z + 1] = Ex[q + nxy];
        ey[z + 1] = Ey[q + nxy];
        ez[z] = Ez[q];
        ex_j[z] = Ex[q + nx];
        ez_j[z] = Ez[q + nx];
        ey_i[z] = Ey[q + 1];
        ez_i[z] = Ez[q + 1];
#pragma unroll
        for (int m = 0; m < 3; m++) h[z][m] = a.f[3 + m][q];
        if (SLAB) flat_psi_load<1>(p[z], a, i, j, kz, ij, nxy);
    }
#pragma unroll
    for (int z = 0; z < Z; z++) {
        if (k + z >= k1) break;
        const cell_t q = q0 + nxy * (cell_t)z;
        const float dEz_dy = ez_j[z] - ez[z], dEy_dz = ey[z + 1] - ey[z], dEx_dz = ex[z + 1] - ex[z];
        const float dEz_dx = ez_i[z] - ez[z], dEy_dx = ey_i[z] - ey[z], dEx_dy = ex_j[z] - ex[z];
        float c[3];
        if (SLAB) {
            flat_psi_curl<1>(p[z], a, i, j, k + z, dEz_dy, dEy_dz, dEx_dz, dEz_dx, dEy_dx, dEx_dy, c);
        } else {
            c[0] = dEz_dy - dEy_dz;
            c[1] = dEx_dz - dEz_dx;
            c[2] = dEy_dx - dEx_dy;
        }
        if (a.src.n) {
            const float *sp = flat_src(a.src, k + z);
            if (sp) {
#pragma unroll
                for (int m = 0; m < 3; m++) c[m] += a.dx * sp[(cell_t)(3 + m) * nxy + ij];
            }
        }
#pragma unroll
        for (int m = 0; m < 3; m++) a.f[3 + m][q] = h[z][m] - a.hb * c[m];
    }
}

template <bool E, bool CPML, bool LOSSY, bool ONE>
__global__ void __launch_bounds__(kFlatThreads) k_flat(const __grid_constant__ FlatArgs a, const __grid_constant__ FlatRange f)
{
    // programmatic dependent launch, as the other step kernels
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // H goes backwards: it starts where E left off, and E where H did, in L2
    const unsigned block = E ? blockIdx.x : gridDim.x - 1 - blockIdx.x;
    int s = kFlatBox;
    if (CPML)
        while (s > 0 && block < f.r[s].first) s--;
    const FlatRegion r = f.r[s];
    const unsigned b = block - r.first, slot = b / r.per;
    const unsigned t = (b - slot * r.per) * (unsigned)kFlatThreads + threadIdx.x, y = t / (unsigned)r.w;
    if (y >= (unsigned)r.rows) return;
    const int x = (int)(t - y * (unsigned)r.w), j = r.j0 + (int)y;
    if (CPML && s != kFlatBox) {
        const int S = a.L - 1, i = s == kFlatX && x >= S ? a.nx - a.L + x - S : 1 + x, k = r.k0 + (int)slot;
        if (E) flat_E_cells<1, true, LOSSY, ONE>(a, i, j, k, r.k1);
        else flat_H_cells<1, true>(a, i, j, k, r.k1);
    } else {
        const int i = (CPML ? a.L : 1) + x, k = r.k0 + kFlatZ * (int)slot;
        if (E) flat_E_cells<kFlatZ, false, LOSSY, ONE>(a, i, j, k, r.k1);
        else flat_H_cells<kFlatZ, false>(a, i, j, k, r.k1);
    }
}

template <bool CPML> static void launch_flat(const cudaLaunchConfig_t &cfg, const FlatArgs &a, const FlatRange &f)
{
    const bool lossy = a.ca[0] != nullptr, one = a.cb[1] == a.cb[0];
    auto E = lossy ? (one ? k_flat<true, CPML, true, true> : k_flat<true, CPML, true, false>)
                   : (one ? k_flat<true, CPML, false, true> : k_flat<true, CPML, false, false>);
    cudaLaunchKernelEx(&cfg, E, a, f);
    cudaLaunchKernelEx(&cfg, k_flat<false, CPML, false, false>, a, f);
}

void launch_flat_step(const FlatArgs &a, cudaStream_t st)
{
    const int L = std::max(1, a.L), nx = a.nx, ny = a.ny, nz = a.nz;
    if (nx < 3 || ny < 3 || nz < 3) return;
    FlatRange f{};
    const int w[kFlatRegions] = {nx - 2, nx - 2, nx - 2, nx - 2, 2 * L - 2, nx - 2 * L};
    const int j0[kFlatRegions] = {1, 1, 1, ny - L, L, L}, j1[kFlatRegions] = {ny - 1, ny - 1, L, ny - 1, ny - L, ny - L};
    const int k0[kFlatRegions] = {1, nz - L, L, L, L, L}, k1[kFlatRegions] = {L, nz - 1, nz - L, nz - L, nz - L, nz - L};
    unsigned blocks = 0;
    for (int s = 0; s < kFlatRegions; s++) {
        const int rows = std::max(0, j1[s] - j0[s]), planes = std::max(0, k1[s] - k0[s]);
        f.r[s] = FlatRegion{blocks, 1, std::max(1, w[s]), j0[s], rows, k0[s], k1[s]};
        if (rows == 0 || planes == 0 || w[s] <= 0) continue;
        f.r[s].per = (unsigned)(((long long)w[s] * rows + kFlatThreads - 1) / kFlatThreads);
        blocks += f.r[s].per * (unsigned)(s == kFlatBox ? (planes + kFlatZ - 1) / kFlatZ : planes);
    }
    if (blocks == 0) return;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kFlatThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    note_launch(2);
    if (a.L > 0) launch_flat<true>(cfg, a, f);
    else launch_flat<false>(cfg, a, f);
}

}  // namespace fdtd
