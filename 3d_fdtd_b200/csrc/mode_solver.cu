// mode_solver.cu -- waveguide eigenmodes on the GPU in FP64: the reference's
// restarted Arnoldi iteration on the beta^2 operator (mode.c:3461-3616).
//
// A `mode` holds 6 complex components per cell of the cross-section, index
// 6*(i + mi*j) + m, m = Ex Ey Ez Hx Hy Hz, with complex ep, mu (3 per cell)
// and PML stretch factors sx, sy (2 per cell).  The solver looks for the mode
// with the largest real beta^2.  Per restart:
//   orthogonalise psi against previous modes (H inner product), boundary
//   condition, optional lateral symmetrisation, zero the PML cells; Krylov
//   basis k_0 = psi/|psi|, k_i = B k_{i-1} with modified Gram-Schmidt into an
//   upper Hessenberg H; the eigenvalue of H with the largest real part, its
//   eigenvector y; psi = sum_j y_j k_j; n_eff = sqrt(lambda)/omega.
// It stops when |n_eff| changes by less than tol, then forms Hz from
// div B = 0 and E from curl H and H-normalises the mode.
//
// Inside the loop only Hx and Hy matter: the operator reads and writes only
// them, the inner products use only them, Hz stays zero and E is recomputed
// from H before any use.  So the device vectors hold (Hx, Hy) per cell and
// the other four components are formed once at the end.
//
// Device arithmetic uses the reference's complex formulas (complex.c:75-149)
// with round-to-nearest intrinsics and no FMA, so one operator application
// equals mode_apply_beta_squared_operator (mode.c:2796-2943) bit for bit.
// Inner products are FP64 tree sums (the reference sums sequentially).  The
// small eigenproblem runs on the host: shifted QR on the Hessenberg matrix for
// the eigenvalues (the reference runs Householder QL sweeps to a 1e-3
// off-diagonal ratio, matrix.c:672-871), and the eigenvector from the
// reference's bordered system (matrix.c:1114-1158): H - lambda I with its
// last row replaced by ones, right-hand side n e_n.  The reference stores the
// last Arnoldi norm one element past its size x size matrix
// (mode.c:3542-3544 with i = size); that value is never read and is not kept.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "common.cuh"
#include "engine.h"
#include "host_ref.h"

namespace fdtd {

using cd = std::complex<double>;

// ---- device complex arithmetic (complex.c), no FMA -------------------------
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(dadd(a.x, b.x), dadd(a.y, b.y)); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(dsub(a.x, b.x), dsub(a.y, b.y)); }
__device__ __forceinline__ double2 csmul(double s, double2 a) { return make_double2(dmul(s, a.x), dmul(s, a.y)); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
    return make_double2(dsub(dmul(a.x, b.x), dmul(a.y, b.y)), dadd(dmul(a.x, b.y), dmul(a.y, b.x)));
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double cmag(double2 a) { return __dsqrt_rn(dadd(dmul(a.x, a.x), dmul(a.y, a.y))); }
__device__ __forceinline__ double2 cdiv(double2 x, double2 y)
{
    const double2 num = cmul(x, cconj(y));
    const double m = cmag(y);
    return csmul(__ddiv_rn(1.0, dmul(m, m)), num);
}
__device__ __forceinline__ double2 crecip(double2 x) { return cdiv(make_double2(1.0, 0.0), x); }

// material and PML of the cross-section, reference layout
struct MsGeom {
    int mi, mj;
    double disc, omega2;
    const double2 *ep, *mu, *pml;   // 3, 3, 2 per cell
    const double2 *inv_epz, *inv_muz; // 1 per cell
    const double *inv_s2;             // 2 per cell: 1 / |sx|^2, 1 / |sy|^2
};

// per-cell 1/ep_z and 1/mu_z (complex_reciprocal), and the real factor of a
// division by sx or sy (cdiv), so that the operator divides by multiplying
__global__ void k_ms_inverses(MsGeom g, double2 *inv_epz, double2 *inv_muz, double *inv_s2)
{
    const int n = g.mi * g.mj;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        inv_epz[c] = crecip(g.ep[3 * c + 2]);
        inv_muz[c] = crecip(g.mu[3 * c + 2]);
        for (int w = 0; w < 2; w++) {
            const double m = cmag(g.pml[2 * c + w]);
            inv_s2[2 * c + w] = __ddiv_rn(1.0, dmul(m, m));
        }
    }
}

// One component of (B in) at cell c (mode.c:2796-2943), w = 0 Hx, 1 Hy; 0 on
// the window edge.  Vectors: v[2c] = Hx, v[2c+1] = Hy.  The two components'
// formulas are each other's with x and y exchanged: n is the neighbour behind
// (left for Hx, below for Hy), q the one ahead across (above, right).  Loads
// go through L2: inside the Krylov kernel other blocks wrote `in`.
__device__ __forceinline__ double2 ms_beta2(const MsGeom &g, const double2 *in, int c, int w)
{
    const int mi = g.mi, mj = g.mj;
    const int i = c % mi, j = c / mi;
    if (i < 1 || i > mi - 2 || j < 1 || j > mj - 2) return make_double2(0.0, 0.0);
    const double d = __ddiv_rn(1.0, g.disc);
    auto H = [&](int cell, int comp) { return __ldcg(in + 2 * cell + comp); };
    auto B = [&](int cell, int comp) { return cmul(g.mu[3 * cell + comp], H(cell, comp)); };
    // cdiv(x, s) of a stretch factor s: x conj(s) / |s|^2
    auto over = [&](double2 x, int cell, int comp) {
        return csmul(g.inv_s2[2 * cell + comp], cmul(x, cconj(g.pml[2 * cell + comp])));
    };
    auto dB = [&](int cell, int comp) {   // dBx/dx or dBy/dy at a cell (forward)
        return over(csmul(d, csub(B(cell + (comp ? mi : 1), comp), B(cell, comp))), cell, comp);
    };
    auto dH = [&](int cell, int comp) {   // dHx/dy or dHy/dx at a cell (backward)
        return over(csmul(d, csub(H(cell, comp), H(cell - (comp ? 1 : mi), comp))), cell, 1 - comp);
    };
    const int n = w ? c - mi : c - 1, q = w ? c + 1 : c + mi;
    const double2 imz = g.inv_muz[c], imz_n = g.inv_muz[n], iez = g.inv_epz[c], iez_q = g.inv_epz[q];
    const double2 e = g.ep[3 * c + 1 - w];
    const double2 t1 = over(csmul(d, csub(cmul(imz, dB(c, 0)), cmul(imz_n, dB(n, 0)))), c, w);
    const double2 t2 = over(csmul(d, csub(cmul(imz, dB(c, 1)), cmul(imz_n, dB(n, 1)))), c, w);
    const double2 t3 = over(cmul(csmul(w ? d : -d, e), csub(cmul(iez_q, dH(q, 1)), cmul(iez, dH(c, 1)))), c, 1 - w);
    const double2 t4 = over(cmul(csmul(w ? -d : d, e), csub(cmul(iez_q, dH(q, 0)), cmul(iez, dH(c, 0)))), c, 1 - w);
    const double2 t5 = csmul(g.omega2, cmul(cmul(e, g.mu[3 * c + w]), H(c, w)));
    return cadd(cadd(cadd(t1, t2), cadd(t3, t4)), t5);
}

__global__ void k_ms_beta2(MsGeom g, const double2 *in, double2 *out)
{
    const int n2 = 2 * g.mi * g.mj;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n2; t += gridDim.x * blockDim.x)
        out[t] = ms_beta2(g, in, t >> 1, t & 1);
}

// ---- inner products: disc^2 * sum conj(a) b over (Hx, Hy) -----------------
// Element t belongs to thread t % (kDotBlocks kDotThreads) of the grid; threads,
// warps and blocks add in a fixed order, whichever kernel does it, so every
// inner product is deterministic.
constexpr int kDotBlocks = 148, kDotThreads = 256;
constexpr int kDotStride = kDotBlocks * kDotThreads;

__device__ __forceinline__ void dot_add(double2 &s, double2 a, double2 b)
{
    s = cadd(s, cmul(cconj(a), b));
}

// sum over the warp in a fixed tree, the same bits in every lane
__device__ __forceinline__ double2 dot_warp(double2 s, int width)
{
    for (int o = width / 2; o > 0; o >>= 1) {
        s.x = dadd(s.x, __shfl_xor_sync(0xffffffffu, s.x, o));
        s.y = dadd(s.y, __shfl_xor_sync(0xffffffffu, s.y, o));
    }
    return s;
}

// the block's sum, in every thread (ws: one value a warp)
__device__ __forceinline__ double2 dot_block(double2 s, double2 *ws)
{
    s = dot_warp(s, 32);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    return dot_warp(ws[threadIdx.x & (kDotThreads / 32 - 1)], kDotThreads / 32);
}
static_assert(kDotBlocks <= kDotThreads, "one thread a block's partial");

// one inner product: the last block to finish (completion count after a fence)
// adds the partials and writes *out (optionally also sqrt(|out|) to *norm_out)
__global__ void __launch_bounds__(kDotThreads) k_ms_dot(const double2 *a, const double2 *b, int n2, double disc2,
                                                      double2 *partials, unsigned *done, double2 *out,
                                                      double *norm_out)
{
    __shared__ double2 ws[2][kDotThreads / 32];
    __shared__ bool last;
    double2 s = make_double2(0.0, 0.0);
    for (int t = blockIdx.x * kDotThreads + threadIdx.x; t < n2; t += kDotStride) dot_add(s, a[t], b[t]);
    s = dot_block(s, ws[0]);
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = s;
        __threadfence();
        last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // every partial fetched at once (one thread walking them took 9 of a dot's 11 us)
    s = threadIdx.x < gridDim.x ? __ldcg(partials + threadIdx.x) : make_double2(0.0, 0.0);
    s = csmul(disc2, dot_block(s, ws[1]));
    if (threadIdx.x == 0) {
        *out = s;
        if (norm_out) *norm_out = __dsqrt_rn(cmag(s));
        *done = 0u;
    }
}

// ---- one Krylov cycle in one cooperative launch ----------------------------
// k_i = B k_{i-1} for i = 1..K with modified Gram-Schmidt,
//   h_j = <k_j, y - sum_{l<j} h_l k_l>,  y = B k_{i-1}.
//
// What bounds it: as kernels a cycle was 470 launches of 2 to 11 us, each
// waiting for the one before (K = 20, 200 x 160 window: 4.3 ms a cycle, the
// arithmetic a few percent of it).  In one launch, with y in registers and the
// basis in L2, each of the K (K + 1) / 2 + K inner products still costs a
// round trip of the grid through L2, 2 x 1.4 us between the two dies: 0.95 ms a
// cycle.  So the products of a step are taken together (low-synchronisation
// Gram-Schmidt, Swirydowicz, Langou, Ananthan, Yang, Thomas, 2021): with
// s_j = <k_j, y> and the Gram matrix G_jl = <k_j, k_l>, whose row i - 1 rides
// along in the same pass, the h above solve (I + strict lower triangle of G)
// h = s, the same numbers to rounding.  A step is then two reductions (h,
// norm) and a barrier: 0.35 ms a cycle, of which 0.15 are its 100 hops.
//
// Reductions: a block's partial sums, one word pair a value, go to the block
// that adds that value up, and the sums to every block.  A word is 16 bytes, a
// double and the reduction's number, written and read whole; the reader polls
// the words themselves, so a hop is one write and one read and needs no fence.
// (A counting barrier and reading the partials after it took as long as both
// hops; every block reading every partial sent 44,000 reads to 37 cache
// lines, slower than the second hop.)  Words are reused by the next reduction:
// a block writes its partials only after it read every sum of this one, and
// the sums were written after every partial was read.
//
// EPT elements of y a thread stay in registers; EPT = 0 keeps y in memory, for
// windows over 75,000 cells.  The blocks are co-resident (cooperative
// launch).  A wait longer than wait_ns sets *err; every later wait sees it and
// the launch ends.
struct MsKrylov {
    MsGeom g;
    double2 *basis;      // K + 1 vectors; k_0 given
    int K, confinement;
    double disc2;
    double2 *H;          // K x K row-major: column i - 1 of step i
    double *norm;        // norm[i] = |k_i|
    ulonglong2 *words;   // partials [value][block](re, im), then sums [value] kWordStride apart; zero at launch
    unsigned *bar;       // zero at launch
    int *err;
    double2 *gram;       // K x K, when it does not fit the blocks' shared memory
    unsigned long long wait_ns;
};
constexpr int kWordStride = 8;   // a sum's words on a cache line of their own: every block polls them

__device__ __forceinline__ unsigned long long ms_clock()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// polls done() until it holds; false when the wait gave up (here or elsewhere)
template <typename F> __device__ __forceinline__ bool ms_poll(const MsKrylov &a, F done)
{
    unsigned long long t0 = 0;
    for (unsigned tries = 1; !done(); tries++) {
        if (tries % 64) continue;
        if (*(volatile int *)a.err) return false;
        const unsigned long long now = ms_clock();
        if (!t0) t0 = now;
        else if (now - t0 > a.wait_ns) {
            atomicExch(a.err, 1);
            return false;
        }
    }
    return true;
}

// grid barrier k (1, 2, ...), by one thread of each block
__device__ __forceinline__ bool ms_barrier(const MsKrylov &a, unsigned k)
{
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
    const unsigned target = k * gridDim.x;
    return ms_poll(a, [&]() {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.bar) : "memory");
        return v >= target;
    });
}

// a 16-byte word (value, number of its inner product), written and read whole
__device__ __forceinline__ void ms_publish(ulonglong2 *w, double v, unsigned long long n)
{
    asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}\n" ::"l"(w),
                 "l"((unsigned long long)__double_as_longlong(v)), "l"(n)
                 : "memory");
}
__device__ __forceinline__ bool ms_read(const ulonglong2 *w, unsigned long long n, double &v)
{
    unsigned long long lo, hi;
    asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}\n"
                 : "=l"(lo), "=l"(hi)
                 : "l"(w)
                 : "memory");
    v = __longlong_as_double((long long)lo);
    return hi == n;
}

// the sum of s over the warp to w[0] (every lane calls it)
__device__ __forceinline__ void warp_sum_to(double2 *w, double2 s)
{
    s = dot_warp(s, 32);
    if ((threadIdx.x & 31) == 0) *w = s;
}

constexpr int kDotWarps = kDotThreads / 32;
__host__ __device__ constexpr size_t ms_shared(int K, bool gram)
{
    return ((size_t)(kDotWarps + 1) * 2 * K + (gram ? (size_t)K * K : 0)) * sizeof(double2);
}

template <int EPT> __global__ void __launch_bounds__(kDotThreads) k_ms_krylov(MsKrylov a)
{
    extern __shared__ __align__(16) double2 dyn[];
    __shared__ double2 ws[2][kDotWarps];
    __shared__ int ok;
    const int n2 = 2 * a.g.mi * a.g.mj, tid = threadIdx.x, nb = gridDim.x, K = a.K;
    const int warp = tid >> 5, lane = tid & 31;
    const int t0 = blockIdx.x * kDotThreads + tid;
    constexpr int R = EPT > 0 ? EPT : 1;
    double2 *wsum = dyn;                         // [warp][2K]: the warps' sums of a reduction
    double2 *sums = dyn + kDotWarps * 2 * K;     // [2K]: its result
    double2 *G = a.gram ? a.gram : sums + 2 * K;   // <k_row, k_col> at [col][row]
    ulonglong2 *part = a.words, *total = a.words + (size_t)4 * K * kDotBlocks;
    double2 yr[R], qr[R];       // y and k_{i-1}
    unsigned nbar = 0, nred = 0;
    double2 *ym = nullptr;      // EPT = 0: y in memory
    // f(element, slot, its value) for this thread's elements, in order
    auto each = [&](auto f) {
        if constexpr (EPT > 0) {
#pragma unroll
            for (int e = 0; e < R; e++)
                if (t0 + e * kDotStride < n2) f(t0 + e * kDotStride, e, yr[e]);
        } else {
            for (int t = t0; t < n2; t += kDotStride) f(t, 0, ym[t]);
        }
    };
    // sums[0..m) = the grid's sums of wsum[.][0..m); false when a wait gave up
    auto reduce = [&](int m) -> bool {
        nred++;
        __syncthreads();
        for (int v = tid; v < m; v += kDotThreads) {
            double2 s = wsum[v];
            for (int w = 1; w < kDotWarps; w++) s = cadd(s, wsum[w * 2 * K + v]);
            ulonglong2 *p = part + 2 * ((size_t)v * kDotBlocks + blockIdx.x);
            ms_publish(p, s.x, nred);
            ms_publish(p + 1, s.y, nred);
        }
        bool good = true;
        for (int v = blockIdx.x, q = 0; v < m; v += nb, q ^= 1) {   // values this block adds up
            double2 s = make_double2(0.0, 0.0);
            if (tid < nb) {
                const ulonglong2 *p = part + 2 * ((size_t)v * kDotBlocks + tid);
                good = ms_poll(a, [&]() {
                    const bool re = ms_read(p, nred, s.x), im = ms_read(p + 1, nred, s.y);
                    return re && im;
                }) && good;
            }
            s = csmul(a.disc2, dot_block(s, ws[q]));
            if (tid < 2) ms_publish(total + v * kWordStride + tid, tid ? s.y : s.x, nred);
        }
        for (int u = tid; u < 2 * m && good; u += kDotThreads) {
            double x = 0.0;
            good = ms_poll(a, [&]() { return ms_read(total + (u >> 1) * kWordStride + (u & 1), nred, x); });
            reinterpret_cast<double *>(sums)[u] = x;
        }
        return !__syncthreads_or(!good);
    };
    for (int i = 1; i <= K; i++) {
        const double2 *prev = a.basis + (size_t)(i - 1) * n2;
        ym = a.basis + (size_t)i * n2;
        each([&](int t, int e, double2 &y) {
            int c = t >> 1;
            if (a.confinement == 1) {   // columns 0 and mi-1 copy their neighbours
                const int x = c % a.g.mi;
                c += x == 0 ? 1 : (x == a.g.mi - 1 ? -1 : 0);
            }
            y = ms_beta2(a.g, prev, c, t & 1);
            if (EPT > 0) qr[e] = prev[t];
        });
        // s_l = <k_l, y> and row i - 1 of G, every l < i in one pass
#pragma unroll 4
        for (int l = 0; l < i; l++) {
            const double2 *q = a.basis + (size_t)l * n2;
            double2 s = make_double2(0.0, 0.0), gs = s;
            each([&](int t, int e, double2 &y) {
                const double2 x = q[t];
                dot_add(s, x, y);
                dot_add(gs, EPT > 0 ? qr[e] : prev[t], x);
            });
            warp_sum_to(wsum + warp * 2 * K + l, s);
            if (l + 1 < i) warp_sum_to(wsum + warp * 2 * K + i + l, gs);
        }
        if (!reduce(2 * i - 1)) return;
        // in device memory it is the grid's: block 0 writes it, the others take this step's
        // row from their sums and the rows before from there, a grid barrier later
        if (!a.gram || blockIdx.x == 0)
            for (int l = tid; l + 1 < i; l += kDotThreads) G[(size_t)l * K + (i - 1)] = sums[i + l];
        __syncthreads();
        auto gram = [&](int row, int col) {
            if (!a.gram) return G[(size_t)col * K + row];
            return row == i - 1 ? sums[i + col] : __ldcg(G + (size_t)col * K + row);
        };
        // h from (I + strictly lower G) h = s, in place, by one warp
        if (warp == 0) {
            if (K <= 32) {
                double2 h = lane < i ? sums[lane] : make_double2(0.0, 0.0);
                for (int j = 0; j + 1 < i; j++) {
                    const double2 hj = make_double2(__shfl_sync(0xffffffffu, h.x, j), __shfl_sync(0xffffffffu, h.y, j));
                    if (lane > j && lane < i) h = csub(h, cmul(hj, gram(lane, j)));
                }
                if (lane < i) sums[lane] = h;
            } else {
                for (int j = 0; j + 1 < i; j++) {
                    const double2 hj = sums[j];
                    for (int k = j + 1 + lane; k < i; k += 32) sums[k] = csub(sums[k], cmul(hj, gram(k, j)));
                    __syncwarp();
                }
            }
        }
        __syncthreads();
        if (blockIdx.x == 0)
            for (int j = tid; j < i; j += kDotThreads) a.H[(size_t)j * K + (i - 1)] = sums[j];
        if (i == K) break;
#pragma unroll 4
        for (int l = 0; l < i; l++) {
            const double2 h = sums[l], *q = a.basis + (size_t)l * n2;
            each([&](int t, int, double2 &y) { y = csub(y, cmul(h, q[t])); });
        }
        double2 s = make_double2(0.0, 0.0);
        each([&](int, int, double2 &y) { dot_add(s, y, y); });
        warp_sum_to(wsum + warp * 2 * K, s);
        if (!reduce(1)) return;
        const double norm = __dsqrt_rn(cmag(sums[0]));
        if (t0 == 0) a.norm[i] = norm;
        const double inv = __ddiv_rn(1.0, norm);
        each([&](int t, int, double2 &y) {
            y = csmul(inv, y);
            if (EPT > 0) a.basis[(size_t)i * n2 + t] = y;
        });
        // the next application reads its neighbours' elements
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            ok = ms_barrier(a, ++nbar);
        }
        __syncthreads();
        if (!ok) return;
    }
}

// the cycle's grid barrier with one arrival of two (fdtd_wait_selftest)
__global__ void k_ms_wait_selftest(MsKrylov a, unsigned long long *elapsed_ns)
{
    const unsigned long long t0 = ms_clock();
    ms_barrier(a, 2);
    *elapsed_ns = ms_clock() - t0;
}

// y -= (*coef) x
__global__ void k_ms_axpy(double2 *y, const double2 *x, const double2 *coef, int n2)
{
    const double2 c = *coef;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n2; t += gridDim.x * blockDim.x)
        y[t] = csub(y[t], cmul(c, x[t]));
}

// y *= 1 / *norm (mode_H_normalize: divisor = 1/norm)
__global__ void k_ms_scale(double2 *y, const double *norm, int n2)
{
    const double s = 1.0 / *norm;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n2; t += gridDim.x * blockDim.x) y[t] = csmul(s, y[t]);
}

// boundary condition (mode.c:1381-1632): confinement 2 zeroes the window edge;
// confinement 1 zeroes rows 0 and mj-1 (columns 1..mi-2) and copies the
// neighbour column into columns 0 and mi-1 (every row)
__global__ void k_ms_bc(double2 *v, int mi, int mj, int confinement)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const double2 z = make_double2(0.0, 0.0);
    if (confinement == 2) {
        // left/right columns (all rows), then top/bottom rows (inner columns)
        if (t < mj) {
            const int cr = (t + 1) * mi - 1, cl = t * mi;
            v[2 * cr] = z; v[2 * cr + 1] = z;
            v[2 * cl] = z; v[2 * cl + 1] = z;
        }
        if (t >= 1 && t < mi - 1) {
            const int ct = t + (mj - 1) * mi, cb = t;
            v[2 * ct] = z; v[2 * ct + 1] = z;
            v[2 * cb] = z; v[2 * cb + 1] = z;
        }
    }
}

// confinement 1 in two ordered launches: vertical zero first, then the
// horizontal zero-gradient copy (which reads the already-zeroed rows)
__global__ void k_ms_bc1_vertical(double2 *v, int mi, int mj)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 1 && t < mi - 1) {
        const double2 z = make_double2(0.0, 0.0);
        const int ct = t + (mj - 1) * mi, cb = t;
        v[2 * ct] = z; v[2 * ct + 1] = z;
        v[2 * cb] = z; v[2 * cb + 1] = z;
    }
}

__global__ void k_ms_bc1_horizontal(double2 *v, int mi, int mj)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < mj) {
        const int cr = (t + 1) * mi - 1, cl = t * mi;
        v[2 * cr] = v[2 * (cr - 1)]; v[2 * cr + 1] = v[2 * (cr - 1) + 1];
        v[2 * cl] = v[2 * (cl + 1)]; v[2 * cl + 1] = v[2 * (cl + 1) + 1];
    }
}

// zero the cells whose PML stretch has an imaginary part (mode.c:1587-1612)
__global__ void k_ms_zero_pml(double2 *v, const double2 *pml, int n)
{
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        if (pml[2 * c].y > 1e-9 || pml[2 * c + 1].y > 1e-9) {
            v[2 * c] = make_double2(0.0, 0.0);
            v[2 * c + 1] = make_double2(0.0, 0.0);
        }
    }
}

// reflection x -> mi-1-x with Hx -> -Hx (mode.c:4494-4527)
__global__ void k_ms_reflect(const double2 *v, double2 *r, int mi, int mj)
{
    const int n = mi * mj;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        const int i = c % mi, j = c / mi;
        const int s = (mi - 1 - i) + j * mi;
        r[2 * s] = csub(make_double2(0.0, 0.0), v[2 * c]);
        r[2 * s + 1] = v[2 * c + 1];
    }
}

// v += (+1 or -1 by the sign of Re *ip) r
__global__ void k_ms_symmetrise(double2 *v, const double2 *r, const double2 *ip, int n2)
{
    const double2 s = make_double2(ip->x > 0 ? 1.0 : -1.0, 0.0);
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n2; t += gridDim.x * blockDim.x)
        v[t] = cadd(v[t], cmul(s, r[t]));
}

// psi = sum_j y_j k_j, j = 0..m-1 in order (k_j at basis + j*n2)
__global__ void k_ms_combine(double2 *psi, const double2 *basis, const double2 *y, int m, int n2)
{
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n2; t += gridDim.x * blockDim.x) {
        double2 s = make_double2(0.0, 0.0);
        for (int j = 0; j < m; j++) s = cadd(s, cmul(y[j], basis[(long long)j * n2 + t]));
        psi[t] = s;
    }
}

// final fields in the reference layout: Hx, Hy from v; Hz = -i/beta (dBx/dx +
// dBy/dy) on interior cells (mode.c:3350-3395); then the boundary condition;
// then E = (-i/omega) ep^-1 curl H on interior cells (mode.c:2330-2397)
__global__ void k_ms_fields_h(MsGeom g, const double2 *v, double2 *f, double2 beta)
{
    const int mi = g.mi, mj = g.mj, n = mi * mj;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        double2 *o = f + 6 * c;
        o[3] = v[2 * c];
        o[4] = v[2 * c + 1];
        o[0] = o[1] = o[2] = o[5] = make_double2(0.0, 0.0);
    }
}

__global__ void k_ms_hz(MsGeom g, double2 *f, double2 beta)
{
    const int mi = g.mi, mj = g.mj, n = mi * mj;
    const double d = 1.0 / g.disc;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        const int i = c % mi, j = c / mi;
        if (i < 1 || i > mi - 2 || j < 1 || j > mj - 2) continue;
        const int r = c + 1, u = c + mi;
        const double2 Bx = cmul(g.mu[3 * c], f[6 * c + 3]), By = cmul(g.mu[3 * c + 1], f[6 * c + 4]);
        const double2 Bx_r = cmul(g.mu[3 * r], f[6 * r + 3]), By_u = cmul(g.mu[3 * u + 1], f[6 * u + 4]);
        const double2 Bx_dx = cdiv(csmul(d, csub(Bx_r, Bx)), g.pml[2 * c]);
        const double2 By_dy = cdiv(csmul(d, csub(By_u, By)), g.pml[2 * c + 1]);
        f[6 * c + 5] = cmul(cdiv(make_double2(0.0, -1.0), beta), cadd(Bx_dx, By_dy));
    }
}

// boundary condition on all 6 components of the final fields
__global__ void k_ms_bc_full(double2 *f, int mi, int mj, int confinement, int pass)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const double2 z = make_double2(0.0, 0.0);
    if (confinement == 2) {
        if (t < mj) {
            const int cr = (t + 1) * mi - 1, cl = t * mi;
            for (int m = 0; m < 6; m++) { f[6 * cr + m] = z; f[6 * cl + m] = z; }
        }
        if (t >= 1 && t < mi - 1) {
            const int ct = t + (mj - 1) * mi, cb = t;
            for (int m = 0; m < 6; m++) { f[6 * ct + m] = z; f[6 * cb + m] = z; }
        }
    } else if (pass == 0) {
        if (t >= 1 && t < mi - 1) {
            const int ct = t + (mj - 1) * mi, cb = t;
            for (int m = 0; m < 6; m++) { f[6 * ct + m] = z; f[6 * cb + m] = z; }
        }
    } else {
        if (t < mj) {
            const int cr = (t + 1) * mi - 1, cl = t * mi;
            for (int m = 0; m < 6; m++) { f[6 * cr + m] = f[6 * (cr - 1) + m]; f[6 * cl + m] = f[6 * (cl + 1) + m]; }
        }
    }
}

__global__ void k_ms_e(MsGeom g, double2 *f, double2 beta, double omega)
{
    const int mi = g.mi, mj = g.mj, n = mi * mj;
    const double d = 1.0 / g.disc;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        const int i = c % mi, j = c / mi;
        if (i < 1 || i > mi - 2 || j < 1 || j > mj - 2) continue;
        const int l = c - 1, dn = c - mi;
        const double2 Hx = f[6 * c + 3], Hy = f[6 * c + 4], Hz = f[6 * c + 5];
        const double2 Hy_l = f[6 * l + 4], Hz_l = f[6 * l + 5];
        const double2 Hx_d = f[6 * dn + 3], Hz_d = f[6 * dn + 5];
        const double2 sx = g.pml[2 * c], sy = g.pml[2 * c + 1];
        const double2 dx_Hy = cdiv(csmul(d, csub(Hy, Hy_l)), sx);
        const double2 dx_Hz = cdiv(csmul(d, csub(Hz, Hz_l)), sx);
        const double2 dy_Hx = cdiv(csmul(d, csub(Hx, Hx_d)), sy);
        const double2 dy_Hz = cdiv(csmul(d, csub(Hz, Hz_d)), sy);
        const double2 iex = crecip(g.ep[3 * c]), iey = crecip(g.ep[3 * c + 1]), iez = g.inv_epz[c];
        const double2 mi_om = csmul(1.0 / omega, make_double2(0.0, -1.0));
        const double2 ib = cmul(make_double2(0.0, 1.0), beta);
        f[6 * c + 0] = cmul(mi_om, cmul(iex, cadd(dy_Hz, cmul(ib, Hy))));
        f[6 * c + 1] = cmul(mi_om, csmul(-1.0, cmul(iey, cadd(dx_Hz, cmul(ib, Hx)))));
        f[6 * c + 2] = cmul(mi_om, cmul(iez, csub(dx_Hy, dy_Hx)));
    }
}

// final H normalisation over all 6 components by 1/|H| (mode_H_normalize)
__global__ void k_ms_scale_full(double2 *f, const double *norm, int n6)
{
    const double s = 1.0 / *norm;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n6; t += gridDim.x * blockDim.x) f[t] = csmul(s, f[t]);
}

// H inner product over the Hx, Hy entries of 6-component fields: gather them first
__global__ void k_ms_gather_h(const double2 *f, double2 *v, int n)
{
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        v[2 * c] = f[6 * c + 3];
        v[2 * c + 1] = f[6 * c + 4];
    }
}

// ============================================================================
// host side
// ============================================================================
namespace {

int grid_blocks(long long n, int threads = 256)
{
    long long b = (n + threads - 1) / threads;
    return (int)(b < 1184 ? (b < 1 ? 1 : b) : 1184);
}

// eigenvalues of an upper Hessenberg complex matrix (row-major n x n) by
// single-shift QR with Wilkinson shifts and deflation (Givens rotations)
bool hessenberg_eigenvalues(std::vector<cd> A, int n, std::vector<cd> &ev)
{
    ev.assign(n, cd(0, 0));
    auto at = [&](int r, int c) -> cd & { return A[(size_t)r * n + c]; };
    int hi = n - 1, iter = 0, total = 0;
    const double eps = 1e-15;
    while (hi >= 0) {
        if (hi == 0) {
            ev[0] = at(0, 0);
            break;
        }
        int l = hi;
        while (l > 0) {
            const double s = std::abs(at(l - 1, l - 1)) + std::abs(at(l, l));
            if (std::abs(at(l, l - 1)) <= eps * (s > 0 ? s : 1.0)) break;
            l--;
        }
        if (l == hi) {
            ev[hi] = at(hi, hi);
            hi--;
            iter = 0;
            continue;
        }
        if (++total > 100000) return false;
        // Wilkinson shift from the trailing 2x2 of the active block
        const cd a = at(hi - 1, hi - 1), b = at(hi - 1, hi), c = at(hi, hi - 1), d = at(hi, hi);
        const cd tr = a + d, det = a * d - b * c;
        const cd disc = std::sqrt(tr * tr / 4.0 - det);
        const cd m1 = tr / 2.0 + disc, m2 = tr / 2.0 - disc;
        cd mu = std::abs(m1 - d) < std::abs(m2 - d) ? m1 : m2;
        if (iter > 0 && iter % 12 == 0) mu = d + std::abs(c);   // exceptional shift
        iter++;
        // QR step on rows/columns l..hi of A - mu I
        for (int k = l; k <= hi; k++) at(k, k) -= mu;
        std::vector<cd> cs(hi - l), sn(hi - l);
        for (int k = l; k < hi; k++) {
            const cd x = at(k, k), y = at(k + 1, k);
            const double r = std::sqrt(std::norm(x) + std::norm(y));
            cd cc = 1.0, ss = 0.0;
            if (r > 0) { cc = x / r; ss = y / r; }
            cs[k - l] = cc; sn[k - l] = ss;
            // rows k, k+1 <- G^H [row k; row k+1]
            for (int col = k; col < n; col++) {
                const cd t1 = at(k, col), t2 = at(k + 1, col);
                at(k, col) = std::conj(cc) * t1 + std::conj(ss) * t2;
                at(k + 1, col) = -ss * t1 + cc * t2;
            }
        }
        for (int k = l; k < hi; k++) {
            const cd cc = cs[k - l], ss = sn[k - l];
            // columns k, k+1 <- [col k, col k+1] G
            for (int row = 0; row <= std::min(k + 2, hi); row++) {
                const cd t1 = at(row, k), t2 = at(row, k + 1);
                at(row, k) = t1 * cc + t2 * ss;
                at(row, k + 1) = -t1 * std::conj(ss) + t2 * std::conj(cc);
            }
        }
        for (int k = l; k <= hi; k++) at(k, k) += mu;
    }
    return true;
}

// solve B x = b (row-major n x n) by Gaussian elimination with partial pivoting
bool linear_solve(std::vector<cd> B, std::vector<cd> b, int n, std::vector<cd> &x)
{
    for (int k = 0; k < n; k++) {
        int p = k;
        for (int r = k + 1; r < n; r++)
            if (std::abs(B[(size_t)r * n + k]) > std::abs(B[(size_t)p * n + k])) p = r;
        if (std::abs(B[(size_t)p * n + k]) == 0.0) return false;
        if (p != k) {
            for (int c = 0; c < n; c++) std::swap(B[(size_t)k * n + c], B[(size_t)p * n + c]);
            std::swap(b[k], b[p]);
        }
        for (int r = k + 1; r < n; r++) {
            const cd f = B[(size_t)r * n + k] / B[(size_t)k * n + k];
            if (f == cd(0, 0)) continue;
            for (int c = k; c < n; c++) B[(size_t)r * n + c] -= f * B[(size_t)k * n + c];
            b[r] -= f * b[k];
        }
    }
    x.assign(n, cd(0, 0));
    for (int r = n - 1; r >= 0; r--) {
        cd s = b[r];
        for (int c = r + 1; c < n; c++) s -= B[(size_t)r * n + c] * x[c];
        x[r] = s / B[(size_t)r * n + r];
    }
    return true;
}

// complex_sqrt of complex.c:151-167 (angle with the 11-digit pi of complex.c,
// exponential by the same power series)
cd reference_sqrt(cd x)
{
    const double pi = 3.14159265359;
    const double mag = std::sqrt(std::sqrt(x.real() * x.real() + x.imag() * x.imag()));
    double angle = std::atan(x.imag() / x.real());
    if (x.real() < 0) angle += pi;
    else if (x.imag() < 0) angle += 2 * pi;
    if (angle > pi) angle -= 2 * pi;
    angle /= 2;
    double re, im;
    cexp_series(angle, &re, &im);
    return cd(mag * re, mag * im);
}

// one allocation handed out in 256-byte aligned pieces
struct Slab {
    char *p = nullptr;
    size_t used = 0;
    ~Slab() { if (p) cudaFree(p); }
    template <typename T> size_t add(size_t count)
    {
        const size_t at = used;
        used = (used + count * sizeof(T) + 255) / 256 * 256;
        return at;
    }
    template <typename T> void at(size_t off, T **out) const { *out = (T *)(p + off); }
};

#define MSK(call)                                      \
    do {                                               \
        if (!cuda_ok((call), #call)) return false;     \
    } while (0)

struct Solver {
    int mi = 0, mj = 0, n = 0, n2 = 0;
    double disc = 0, omega = 0;
    cudaStream_t st = nullptr;
    Slab slab;
    double2 *ep = nullptr, *mu = nullptr, *pml = nullptr, *iez = nullptr, *imz = nullptr;
    double2 *psi = nullptr, *basis = nullptr, *tmp = nullptr, *part = nullptr, *scal = nullptr, *y = nullptr;
    double2 *prev = nullptr, *f = nullptr, *gram = nullptr;
    double *norm = nullptr, *is2 = nullptr;
    unsigned *done = nullptr, *bar = nullptr;
    ulonglong2 *words = nullptr;            // then bar, cleared together
    int *err = nullptr;
    MsGeom g{};

    ~Solver()
    {
        if (st) {
            cudaStreamSynchronize(st);
            cudaStreamDestroy(st);
        }
    }

    // partial and sum words of a cycle of K steps (2K values), then the barrier's count
    static size_t words_count(size_t K) { return 2 * K * (2 * kDotBlocks + kWordStride) + 1; }
    // the Gram matrix fits a block's shared memory
    static bool gram_shared(size_t K) { return ms_shared((int)K, true) <= 200 * 1024; }

    bool setup(const mode &m, double om, int basis_vectors, int nprev)
    {
        mi = m.i; mj = m.j; n = mi * mj; n2 = 2 * n;
        disc = m.disc; omega = om;
        MSK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        const size_t nn = (size_t)n, kv = (size_t)basis_vectors, np = (size_t)(nprev > 0 ? nprev : 1);
        const size_t o_ep = slab.add<double2>(3 * nn), o_mu = slab.add<double2>(3 * nn), o_pml = slab.add<double2>(2 * nn),
                     o_iez = slab.add<double2>(nn), o_imz = slab.add<double2>(nn), o_is2 = slab.add<double>(2 * nn),
                     o_psi = slab.add<double2>(2 * nn), o_basis = slab.add<double2>(kv * 2 * nn),
                     o_tmp = slab.add<double2>(2 * nn), o_part = slab.add<double2>(kDotBlocks),
                     o_words = slab.add<ulonglong2>(words_count(kv - 1)),
                     o_done = slab.add<unsigned>(4), o_scal = slab.add<double2>((kv + 1) * (kv + 1) + 8),
                     o_y = slab.add<double2>(kv + 1), o_prev = slab.add<double2>(np * 2 * nn),
                     o_f = slab.add<double2>(6 * nn),
                     o_gram = slab.add<double2>(gram_shared(kv - 1) ? 0 : (kv - 1) * (kv - 1));
        MSK(cudaMalloc(&slab.p, slab.used));
        slab.at(o_ep, &ep); slab.at(o_mu, &mu); slab.at(o_pml, &pml); slab.at(o_iez, &iez); slab.at(o_imz, &imz);
        slab.at(o_is2, &is2); slab.at(o_psi, &psi); slab.at(o_basis, &basis); slab.at(o_tmp, &tmp);
        slab.at(o_part, &part); slab.at(o_done, &done); slab.at(o_scal, &scal); slab.at(o_y, &y);
        slab.at(o_prev, &prev); slab.at(o_f, &f);
        slab.at(o_words, &words);
        if (!gram_shared(kv - 1)) slab.at(o_gram, &gram);
        bar = (unsigned *)(words + words_count(kv - 1) - 1);
        err = (int *)(done + 2);
        // after the K x K matrix H(r, c) = scal[1 + r K + c]: the norms, read back with it
        norm = (double *)(scal + 1 + (kv - 1) * (kv - 1));
        MSK(cudaMemsetAsync(done, 0, 4 * sizeof(unsigned), st));
        MSK(cudaMemsetAsync(scal, 0, ((kv + 1) * (kv + 1) + 8) * sizeof(double2), st));
        static_assert(sizeof(complex) == sizeof(double2), "complex layout");
        MSK(cudaMemcpyAsync(ep, m.ep.m, 3 * (size_t)n * sizeof(double2), cudaMemcpyHostToDevice, st));
        MSK(cudaMemcpyAsync(mu, m.mu.m, 3 * (size_t)n * sizeof(double2), cudaMemcpyHostToDevice, st));
        MSK(cudaMemcpyAsync(pml, m.pml.m, 2 * (size_t)n * sizeof(double2), cudaMemcpyHostToDevice, st));
        g.mi = mi; g.mj = mj; g.disc = disc; g.omega2 = om * om;
        g.ep = ep; g.mu = mu; g.pml = pml; g.inv_epz = iez; g.inv_muz = imz; g.inv_s2 = is2;
        note_launch();
        k_ms_inverses<<<grid_blocks(n), 256, 0, st>>>(g, iez, imz, is2);
        return cuda_ok(cudaGetLastError(), "mode solver setup");
    }

    // *out = <a, b>_H (and *nrm = sqrt|<a,b>| when nrm)
    void dot(const double2 *a, const double2 *b, double2 *out, double *nrm)
    {
        note_launch();
        k_ms_dot<<<kDotBlocks, kDotThreads, 0, st>>>(a, b, n2, disc * disc, part, done, out, nrm);
    }
    void axpy(double2 *v, const double2 *x, const double2 *coef)
    {
        note_launch();
        k_ms_axpy<<<grid_blocks(n2), 256, 0, st>>>(v, x, coef, n2);
    }
    void scale(double2 *v, const double *nrm)
    {
        note_launch();
        k_ms_scale<<<grid_blocks(n2), 256, 0, st>>>(v, nrm, n2);
    }
    void normalize(double2 *v)
    {
        dot(v, v, scal, norm);
        scale(v, norm);
    }
    void bc(double2 *v, int confinement)
    {
        const int len = mi > mj ? mi : mj;
        note_launch();
        if (confinement == 2) {
            k_ms_bc<<<(len + 255) / 256, 256, 0, st>>>(v, mi, mj, 2);
        } else {
            k_ms_bc1_vertical<<<(len + 255) / 256, 256, 0, st>>>(v, mi, mj);
            note_launch();
            k_ms_bc1_horizontal<<<(len + 255) / 256, 256, 0, st>>>(v, mi, mj);
        }
    }
    void apply(const double2 *in, double2 *out)
    {
        note_launch();
        k_ms_beta2<<<grid_blocks(n2), 256, 0, st>>>(g, in, out);
    }
    // k_1..k_K, H and the norms from k_0 (see k_ms_krylov)
    bool krylov(int K, int confinement)
    {
        MsKrylov a{g, basis, K, confinement, disc * disc, scal + 1, norm, words, bar, err, gram, 1000000000ull};
        MSK(cudaMemsetAsync(words, 0, words_count(K) * sizeof(ulonglong2), st));
        const int per = (n2 + kDotStride - 1) / kDotStride;
        const void *fn = per <= 1 ? (const void *)k_ms_krylov<1> : per <= 2 ? (const void *)k_ms_krylov<2>
                         : per <= 4 ? (const void *)k_ms_krylov<4> : (const void *)k_ms_krylov<0>;
        // blocks past the last element would only add zero partials
        const int blocks = std::min(kDotBlocks, (n2 + kDotThreads - 1) / kDotThreads);
        const size_t smem = ms_shared(K, !gram);
        MSK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        void *args[] = {&a};
        note_launch();
        return cuda_ok(cudaLaunchCooperativeKernel(fn, dim3((unsigned)blocks), dim3(kDotThreads), args, smem, st),
                       "Krylov cycle");
    }
};

}  // namespace

void launch_mode_wait_selftest(unsigned long long limit_ns, unsigned *bar, int *err, unsigned long long *elapsed_ns,
                               cudaStream_t st)
{
    MsKrylov a{};
    a.bar = bar;
    a.err = err;
    a.wait_ns = limit_ns;
    note_launch();
    k_ms_wait_selftest<<<1, 1, 0, st>>>(a, elapsed_ns);
}

bool mode_apply_beta2_device(const mode &in, double omega, mode &out)
{
    Solver s;
    if (!s.setup(in, omega, 1, 0)) return false;
    std::vector<double2> h((size_t)s.n2);
    for (int c = 0; c < s.n; c++) {
        h[2 * c] = make_double2(in.fields.m[6 * c + 3].re, in.fields.m[6 * c + 3].im);
        h[2 * c + 1] = make_double2(in.fields.m[6 * c + 4].re, in.fields.m[6 * c + 4].im);
    }
    MSK(cudaMemcpyAsync(s.psi, h.data(), h.size() * sizeof(double2), cudaMemcpyHostToDevice, s.st));
    s.apply(s.psi, s.tmp);
    MSK(cudaGetLastError());
    MSK(cudaMemcpyAsync(h.data(), s.tmp, h.size() * sizeof(double2), cudaMemcpyDeviceToHost, s.st));
    MSK(cudaStreamSynchronize(s.st));
    for (int c = 0; c < s.n; c++) {
        for (int m = 0; m < 6; m++) out.fields.m[6 * c + m] = complex{0.0, 0.0};
        out.fields.m[6 * c + 3] = complex{h[2 * c].x, h[2 * c].y};
        out.fields.m[6 * c + 4] = complex{h[2 * c + 1].x, h[2 * c + 1].y};
    }
    return true;
}

bool mode_solve_device(mode *psi, double omega, double tol, const mode *prev, int nprev, int size, int confinement,
                       int lateral_symmetry, int max_restarts, cd *beta_out, int *restarts_out)
{
    const int K = size;
    Solver s;
    if (!s.setup(*psi, omega, K + 1, nprev)) return false;
    const int n = s.n, n2 = s.n2;
    // start vector: mode_initialize_rand (mode.c:1192-1206), Hx then Hy per cell
    std::vector<double2> h((size_t)n2);
    for (int c = 0; c < n; c++) {
        h[2 * c] = make_double2((double)rand(), 0.0);
        h[2 * c + 1] = make_double2((double)rand(), 0.0);
    }
    MSK(cudaMemcpyAsync(s.psi, h.data(), h.size() * sizeof(double2), cudaMemcpyHostToDevice, s.st));
    for (int p = 0; p < nprev; p++) {
        for (int c = 0; c < n; c++) {
            h[2 * c] = make_double2(prev[p].fields.m[6 * c + 3].re, prev[p].fields.m[6 * c + 3].im);
            h[2 * c + 1] = make_double2(prev[p].fields.m[6 * c + 4].re, prev[p].fields.m[6 * c + 4].im);
        }
        MSK(cudaMemcpyAsync(s.prev + (size_t)p * n2, h.data(), h.size() * sizeof(double2), cudaMemcpyHostToDevice,
                            s.st));
        MSK(cudaStreamSynchronize(s.st));   // h is reused
    }
    s.normalize(s.psi);   // mode_H_normalize after the random start
    // scalar slots on the device: scal[0] scratch, scal[1 + r*K + c] = H(r, c)
    double2 *Hd = s.scal + 1;
    std::vector<double2> Hh((size_t)K * K);
    std::vector<cd> H((size_t)K * K), ev, yv;
    cd beta(0, 0);
    double n_mag = 100.0, n_diff = 100.0;
    int restarts = 0;
    while (std::fabs(n_diff) > tol) {
        if (restarts >= max_restarts) {
            set_error(FDTD_ERR_TIMEOUT, "mode solver: |n_eff| still changing by %.3g after %d restarts", n_diff,
                      restarts);
            return false;
        }
        // orthogonalise against previous modes (one pass), normalising in between
        s.normalize(s.psi);
        for (int p = nprev - 1; p >= 0; p--) {
            s.dot(s.prev + (size_t)p * n2, s.psi, s.scal, nullptr);
            s.axpy(s.psi, s.prev + (size_t)p * n2, s.scal);
            s.normalize(s.psi);
        }
        s.bc(s.psi, confinement);   // after mode_apply_H_curl, which only changes E
        if (lateral_symmetry) {
            note_launch();
            k_ms_reflect<<<grid_blocks(n), 256, 0, s.st>>>(s.psi, s.tmp, s.mi, s.mj);
            s.dot(s.psi, s.tmp, s.scal, nullptr);
            note_launch();
            k_ms_symmetrise<<<grid_blocks(n2), 256, 0, s.st>>>(s.psi, s.tmp, s.scal, n2);
        }
        note_launch();
        k_ms_zero_pml<<<grid_blocks(n), 256, 0, s.st>>>(s.psi, s.pml, n);
        // Krylov basis k_0..k_K
        double2 *k0 = s.basis;
        MSK(cudaMemcpyAsync(k0, s.psi, (size_t)n2 * sizeof(double2), cudaMemcpyDeviceToDevice, s.st));
        s.normalize(k0);
        s.bc(k0, confinement);
        if (!s.krylov(K, confinement)) return false;
        // H and, right after it, the norms
        std::vector<double2> back((size_t)K * K + (K + 1) / 2);
        MSK(cudaMemcpyAsync(back.data(), Hd, back.size() * sizeof(double2), cudaMemcpyDeviceToHost, s.st));
        int late = 0;
        MSK(cudaMemcpyAsync(&late, s.err, sizeof(int), cudaMemcpyDeviceToHost, s.st));
        MSK(cudaStreamSynchronize(s.st));
        if (late) {
            set_error(FDTD_ERR_TIMEOUT, "mode solver: a device-side wait gave up");
            return false;
        }
        std::copy(back.begin(), back.begin() + (size_t)K * K, Hh.begin());
        const double *sub = (const double *)(back.data() + (size_t)K * K);
        for (int r = 0; r < K; r++)
            for (int c = 0; c < K; c++) H[(size_t)r * K + c] = cd(Hh[(size_t)r * K + c].x, Hh[(size_t)r * K + c].y);
        for (int i = 1; i < K; i++) H[(size_t)i * K + (i - 1)] = cd(sub[i], 0.0);
        // eigenvalue with the largest real part (index 0 unless some real part > 0)
        if (!hessenberg_eigenvalues(H, K, ev)) {
            set_error(FDTD_ERR_CUDA, "mode solver: Hessenberg QR did not converge");
            return false;
        }
        int best = 0;
        double bmax = 0.0;
        for (int i = 0; i < K; i++)
            if (ev[i].real() > bmax) { bmax = ev[i].real(); best = i; }
        const cd lam = ev[best];
        // eigenvector from (H - lambda I) with the last row replaced by ones, rhs n e_n
        std::vector<cd> B(H), rhs((size_t)K, cd(0, 0));
        for (int i = 0; i < K; i++) B[(size_t)i * K + i] -= lam;
        for (int c = 0; c < K; c++) B[(size_t)(K - 1) * K + c] = cd(1, 0);
        rhs[K - 1] = cd((double)K, 0);
        if (!linear_solve(B, rhs, K, yv)) {
            set_error(FDTD_ERR_CUDA, "mode solver: singular eigenvector system");
            return false;
        }
        double yn = 0;
        for (auto &v : yv) yn += std::norm(v);
        yn = std::sqrt(yn);
        std::vector<double2> yd((size_t)K);
        for (int i = 0; i < K; i++) yd[i] = make_double2(yv[i].real() / yn, yv[i].imag() / yn);
        MSK(cudaMemcpyAsync(s.y, yd.data(), yd.size() * sizeof(double2), cudaMemcpyHostToDevice, s.st));
        note_launch();
        k_ms_combine<<<grid_blocks(n2), 256, 0, s.st>>>(s.psi, s.basis, s.y, K, n2);
        MSK(cudaGetLastError());   // yd is pageable: staged when the copy returned
        beta = reference_sqrt(lam);
        const cd n_eff = beta / omega;
        const double n_old = n_mag;
        n_mag = std::abs(n_eff);
        n_diff = n_mag - n_old;
        restarts++;
    }
    // final fields: Hz from div B, boundary, E from curl H, boundary, H-normalise
    const double2 b2 = make_double2(beta.real(), beta.imag());
    note_launch();
    k_ms_fields_h<<<grid_blocks(n), 256, 0, s.st>>>(s.g, s.psi, s.f, b2);
    note_launch();
    k_ms_hz<<<grid_blocks(n), 256, 0, s.st>>>(s.g, s.f, b2);
    const int len = s.mi > s.mj ? s.mi : s.mj;
    for (int pass = 0; pass < (confinement == 2 ? 1 : 2); pass++) {
        note_launch();
        k_ms_bc_full<<<(len + 255) / 256, 256, 0, s.st>>>(s.f, s.mi, s.mj, confinement, pass);
    }
    note_launch();
    k_ms_e<<<grid_blocks(n), 256, 0, s.st>>>(s.g, s.f, b2, omega);
    for (int pass = 0; pass < (confinement == 2 ? 1 : 2); pass++) {
        note_launch();
        k_ms_bc_full<<<(len + 255) / 256, 256, 0, s.st>>>(s.f, s.mi, s.mj, confinement, pass);
    }
    note_launch();
    k_ms_gather_h<<<grid_blocks(n), 256, 0, s.st>>>(s.f, s.tmp, n);
    s.dot(s.tmp, s.tmp, s.scal, s.norm);
    note_launch();
    k_ms_scale_full<<<grid_blocks(6LL * n), 256, 0, s.st>>>(s.f, s.norm, 6 * n);
    MSK(cudaGetLastError());
    MSK(cudaMemcpyAsync(psi->fields.m, s.f, 6 * (size_t)n * sizeof(double2), cudaMemcpyDeviceToHost, s.st));
    MSK(cudaStreamSynchronize(s.st));
    if (beta_out) *beta_out = beta;
    if (restarts_out) *restarts_out = restarts;
    return true;
}

}  // namespace fdtd
