// umma_gemm.cu -- BF16 GEMM on the 5th-generation tensor cores (tcgen05), FP32
// accumulation in tensor memory, fused bias / activation epilogue.  Used by
// the surrogate network (surrogate.cu); the FDTD stencil has no contraction.
//
//   pre[m][n] = alpha * sum_k A[m][k] B[n][k] + beta * C32[m][n] + bias[n]
//   Z32 = pre (optional), post = act(pre) (identity or GELU),
//   C32 = post (optional, FP32), C16 = post (optional, BF16)
// A is M x K and B is N x K, both K-major (row stride lda / ldb elements,
// multiples of 8; K a multiple of 8).  Ragged M, N and K are zero-filled.
//
// One CTA (8 warps) owns a 128 x BN tile of C, BN 32 or 128:
//   warp 0 allocates BN TMEM columns (tcgen05.alloc) for the FP32
//   accumulator (TMEM lane = row of the tile);
//   K tiles of 64 go through a ring of 4 shared-memory stages in the canonical
//   K-major layout without swizzle -- 8-row x 16-byte core matrices, the two
//   8-element K halves of an MMA step 128 B apart (LBO), successive 8-row
//   groups 1024 B apart (SBO).  K-major operands arrive by cp.async, three
//   tiles ahead; an operand stored the other way round (the weight gradient's
//   dZ and H, the backward pass's W) is read as 8 x 8 blocks, transposed in
//   registers and stored as whole core matrices, so no transposed copy of it
//   is ever written to memory;
//   per tile, after a generic-to-async proxy fence and a barrier, one thread
//   issues the tile's tcgen05.mma.cta_group::1.kind::f16 (M 128, N BN, K 16
//   each, four of them) and tcgen05.commit to the stage's mbarrier; a stage is
//   waited for only when it is refilled, three tiles later;
//   epilogue: warps w and w + 4 read TMEM lanes 32 (w % 4)... with tcgen05.ld
//   32x32b.x16, half of the columns each, and store whole rows as float4.
// Waits are bounded in time; a wait that gives up sets *err, waits (bounded)
// for the MMAs in flight, frees the TMEM and returns.
//
// What bounds it: the network's products are tiny (batch 64..512 x 256 x 256),
// so a launch is latency: one K loop's loads, its MMAs and the epilogue.  One
// 256-column tile per CTA with one 32-wide stage put 128 x 256 x 256 on a
// single SM, which then waited for memory and for the MMAs eight times over:
// 48 to 59 us a product.  32-column tiles with everything in flight run on
// eight SMs: 9 to 12 us a launch, of which part is the wait for the previous
// one.  BN is 32 until that fills the chip twice (2 x 148 tiles), then 128,
// which stages A a quarter as often.
// Two products with no order between them (a layer's weight gradient and the
// gradient of its input) and the layer's bias sums share one launch: a training
// step of batch 128 is 11 launches where it was 40, 0.15 ms where it was 0.83
// (host copies included), a prediction and input gradient of 64 rows 0.17 ms
// where they were 0.60.
#include <cuda_bf16.h>

#include "common.cuh"
#include "engine.h"

namespace fdtd {

constexpr int kGemmBM = 128, kGemmBK = 64, kGemmThreads = 256, kGemmStages = 4;
constexpr unsigned kGemmSBO = (kGemmBK / 8) * 128;   // bytes between 8-row groups
constexpr unsigned kGemmLBO = 128;                   // bytes between the two K halves of a step
constexpr unsigned long long kGemmWaitNs = 1000000000ull;

__device__ __forceinline__ unsigned su32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long gtime()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ bool mbar_test(unsigned long long *bar, unsigned parity)
{
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok)
                 : "r"(su32(bar)), "r"(parity)
                 : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool mbar_wait_for(unsigned long long *bar, unsigned parity, unsigned long long ns)
{
    const unsigned long long t0 = gtime();
    for (;;) {
        if (mbar_test(bar, parity)) return true;
        if (gtime() - t0 > ns) return false;
    }
}

// K-major, no swizzle, version 1 (Blackwell) shared-memory matrix descriptor
__device__ __forceinline__ unsigned long long umma_desc(unsigned saddr)
{
    return (unsigned long long)((saddr >> 4) & 0x3FFFu) | ((unsigned long long)((kGemmLBO >> 4) & 0x3FFFu) << 16) |
           ((unsigned long long)((kGemmSBO >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// kind::f16 instruction descriptor: D F32, A and B BF16, both K-major, M 128, N bn
__host__ __device__ constexpr unsigned umma_idesc(int bn)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(bn >> 3) << 17) | ((unsigned)(kGemmBM >> 4) << 24);
}

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }

// derivative of GELU
__device__ __forceinline__ float gelu_grad(float x)
{
    const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
    return cdf + x * pdf;
}

constexpr int kSumCols = 32, kSumRows = 128;   // a column-sum block: 32 columns, staged 128 rows at a time

struct GemmGroup {
    GemmArgs g[2];
    ColSum cs;
    int tiles[2], cols[2];      // CTAs and column tiles of each product
};

// one operand tile (R rows from r0, K from k0) into `dst` by asynchronous copies
template <int R>
__device__ __forceinline__ void stage_rows(unsigned char *dst, const __nv_bfloat16 *P, int ld, int rows, int r0, int k0,
                                           int K)
{
    for (int q = threadIdx.x; q < R * (kGemmBK / 8); q += kGemmThreads) {
        // 8 rows, then 4 chunks, of a 32-lane group: shared addresses run on without bank conflicts
        const int r = (q & 7) | ((q >> 6) << 3), c = (q >> 3) & 7;
        const int gr = r0 + r, gk = k0 + 8 * c;
        const bool in = gr < rows && gk < K;
        const __nv_bfloat16 *src = in ? P + (long long)gr * ld + gk : P;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(su32(dst + (r >> 3) * kGemmSBO + c * 128 +
                                                                                 (r & 7) * 16)),
                     "l"(src), "r"(in ? 16 : 0)
                     : "memory");
    }
}

// the same tile of an operand stored [K][ld] (rows of the tile contiguous): 8 x
// 8 blocks, transposed in registers
template <int R>
__device__ __forceinline__ void stage_rows_t(unsigned char *dst, const __nv_bfloat16 *P, int ld, int rows, int r0,
                                             int k0, int K)
{
    for (int q = threadIdx.x; q < (R / 8) * (kGemmBK / 8); q += kGemmThreads) {
        const int rb = q % (R / 8), c = q / (R / 8);
        const int gr = r0 + 8 * rb, gk = k0 + 8 * c;
        uint4 v[8];
        const bool in = gr < rows && gk < K;
#pragma unroll
        for (int k = 0; k < 8; k++)
            v[k] = in ? *reinterpret_cast<const uint4 *>(P + (long long)(gk + k) * ld + gr) : make_uint4(0, 0, 0, 0);
        uint4 *out = reinterpret_cast<uint4 *>(dst + rb * kGemmSBO + c * 128);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            unsigned w[8];
#pragma unroll
            for (int k = 0; k < 8; k++) w[k] = j == 0 ? v[k].x : j == 1 ? v[k].y : j == 2 ? v[k].z : v[k].w;
            out[2 * j] = make_uint4(__byte_perm(w[0], w[1], 0x5410), __byte_perm(w[2], w[3], 0x5410),
                                    __byte_perm(w[4], w[5], 0x5410), __byte_perm(w[6], w[7], 0x5410));
            out[2 * j + 1] = make_uint4(__byte_perm(w[0], w[1], 0x7632), __byte_perm(w[2], w[3], 0x7632),
                                        __byte_perm(w[4], w[5], 0x7632), __byte_perm(w[6], w[7], 0x7632));
        }
    }
}

template <int BN> constexpr int stage_bytes() { return (kGemmBM + BN) * kGemmBK * 2; }

// rows of 32 columns are staged together (their loads overlap), then one
// thread per column adds them in order
__device__ __forceinline__ void column_sums(const ColSum &cs, int block, float *sm)
{
    const int c0 = block * kSumCols, tid = threadIdx.x;
    float s = 0.0f;
    for (int r0 = 0; r0 < cs.rows; r0 += kSumRows) {
        const int n = min(kSumRows, cs.rows - r0);
        for (int q = tid; q < n * kSumCols; q += kGemmThreads) {
            const int c = c0 + q % kSumCols;
            sm[q] = c < cs.cols ? cs.in[(long long)(r0 + q / kSumCols) * cs.ld + c] : 0.0f;
        }
        __syncthreads();
        if (tid < kSumCols)
            for (int r = 0; r < n; r++) s += sm[r * kSumCols + tid];
        __syncthreads();
    }
    if (tid < kSumCols && c0 + tid < cs.cols) cs.out[c0 + tid] = s;
}

// v[0..16) of one row to dst[0..n): whole float4s where the row allows it
__device__ __forceinline__ void store_row16(float *dst, int n, bool vec, const float (&v)[16])
{
    if (vec && n >= 16) {
#pragma unroll
        for (int i = 0; i < 4; i++)
            reinterpret_cast<float4 *>(dst)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        return;
    }
#pragma unroll
    for (int i = 0; i < 16; i++)
        if (i < n) dst[i] = v[i];
}
__device__ __forceinline__ void load_row16(const float *src, int n, bool vec, float (&v)[16])
{
    if (vec && n >= 16) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float4 t = reinterpret_cast<const float4 *>(src)[i];
            v[4 * i] = t.x; v[4 * i + 1] = t.y; v[4 * i + 2] = t.z; v[4 * i + 3] = t.w;
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = i < n ? src[i] : 0.0f;
}
// a row's 16 values from `col` can move as 16-byte vectors
__device__ __forceinline__ bool vec16(const void *p, int ld_bytes, int col_bytes)
{
    return (((uintptr_t)p | (unsigned)ld_bytes | (unsigned)col_bytes) & 15) == 0;
}

__device__ __forceinline__ void gemm_epilogue16(const GemmArgs &g, int row, int col, const unsigned (&r)[16])
{
    const int n = g.N - col;
    if (row >= g.M || n <= 0) return;
    float v[16], t[16];
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = g.alpha * __uint_as_float(r[i]);
    if (g.beta != 0.0f) {
        const float *c = g.C32 + (long long)row * g.ldc32 + col;
        load_row16(c, n, vec16(g.C32, g.ldc32 * 4, col * 4), t);
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] += g.beta * t[i];
    }
    if (g.bias) {
        load_row16(g.bias + col, n, vec16(g.bias, 0, col * 4), t);
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] += t[i];
    }
    if (g.Z32) store_row16(g.Z32 + (long long)row * g.ldz + col, n, vec16(g.Z32, g.ldz * 4, col * 4), v);
    if (g.act == 1) {
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = gelu(v[i]);
    } else if (g.act == 2) {
        load_row16(g.Zin + (long long)row * g.ldz + col, n, vec16(g.Zin, g.ldz * 4, col * 4), t);
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = v[i] * gelu_grad(t[i]);
    }
    if (g.C32) store_row16(g.C32 + (long long)row * g.ldc32 + col, n, vec16(g.C32, g.ldc32 * 4, col * 4), v);
    if (g.C16) {
        __nv_bfloat16 *c = g.C16 + (long long)row * g.ldc16 + col;
        if (n >= 16 && vec16(g.C16, g.ldc16 * 2, col * 2)) {
            union { __nv_bfloat16 h[16]; uint4 u[2]; } p;
#pragma unroll
            for (int i = 0; i < 16; i++) p.h[i] = __float2bfloat16_rn(v[i]);
            reinterpret_cast<uint4 *>(c)[0] = p.u[0];
            reinterpret_cast<uint4 *>(c)[1] = p.u[1];
        } else {
#pragma unroll
            for (int i = 0; i < 16; i++)
                if (i < n) c[i] = __float2bfloat16_rn(v[i]);
        }
    }
}

template <int BN>
__global__ void __launch_bounds__(kGemmThreads) k_umma_gemm(const __grid_constant__ GemmGroup grp)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) unsigned long long bar[kGemmStages];
    __shared__ unsigned tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int tile = (int)blockIdx.x;
    const bool second = tile >= grp.tiles[0];
    if (second) tile -= grp.tiles[0];
    if (second && tile >= grp.tiles[1]) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        column_sums(grp.cs, tile - grp.tiles[1], reinterpret_cast<float *>(smem));
        return;
    }
    const GemmArgs &g = grp.g[second ? 1 : 0];
    const int nc = grp.cols[second ? 1 : 0];
    const int m0 = (tile / nc) * kGemmBM, n0 = (tile % nc) * BN;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&tmem_base)),
                     "r"((unsigned)BN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0)
        for (int s = 0; s < kGemmStages; s++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(su32(&bar[s])));
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const unsigned tmem = tmem_base;
    // the set-up above may overlap the previous kernel; its results are read from here on
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int ktiles = (g.K + kGemmBK - 1) / kGemmBK;
    auto load = [&](int kt) {
        unsigned char *sA = smem + (kt % kGemmStages) * stage_bytes<BN>(), *sB = sA + kGemmBM * kGemmBK * 2;
        const int k0 = kt * kGemmBK;
        if (g.a_t) stage_rows_t<kGemmBM>(sA, g.A, g.lda, g.M, m0, k0, g.K);
        else stage_rows<kGemmBM>(sA, g.A, g.lda, g.M, m0, k0, g.K);
        if (g.b_t) stage_rows_t<BN>(sB, g.B, g.ldb, g.N, n0, k0, g.K);
        else stage_rows<BN>(sB, g.B, g.ldb, g.N, n0, k0, g.K);
    };
    auto parity = [](int kt) { return (unsigned)(kt / kGemmStages) & 1u; };
    for (int kt = 0; kt < kGemmStages - 1; kt++) {
        if (kt < ktiles) load(kt);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    int issued = 0;    // tiles whose MMAs were issued
    bool failed = false;
    for (int kt = 0; kt < ktiles; kt++) {
        // refill the previous tile's stage, once its MMAs have read it
        const int nk = kt + kGemmStages - 1;
        bool late = false;
        if (nk < ktiles) {
            if (kt > 0) late = !mbar_wait_for(&bar[(kt - 1) % kGemmStages], parity(kt - 1), kGemmWaitNs);
            if (!late) load(nk);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kGemmStages - 1) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        failed = __syncthreads_or(late);
        if (failed) break;
        if (tid == 0) {
            const unsigned sA = su32(smem + (kt % kGemmStages) * stage_bytes<BN>()), sB = sA + kGemmBM * kGemmBK * 2;
            const int steps = min(kGemmBK, g.K - kt * kGemmBK + 15) / 16;
            asm volatile("tcgen05.fence::after_thread_sync;");
            for (int s = 0; s < steps; s++) {
                const unsigned long long da = umma_desc(sA + s * 256), db = umma_desc(sB + s * 256);
                const unsigned acc = (kt > 0 || s > 0) ? 1u : 0u;
                asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                             " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
                             "l"(da), "l"(db), "r"(umma_idesc(BN)), "r"(acc));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             su32(&bar[kt % kGemmStages]))
                         : "memory");
        }
        issued = kt + 1;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    // the last commit covers every MMA before it
    if (issued > 0) {
        const bool done = mbar_wait_for(&bar[(issued - 1) % kGemmStages], parity(issued - 1), kGemmWaitNs);
        failed = __syncthreads_or(failed || !done);
    }
    if (failed) {
        if (tid == 0) atomicExch(g.err, 1);
    } else {
        asm volatile("tcgen05.fence::after_thread_sync;");
        const int quad = warp & 3, half = warp >> 2;
        const int row = m0 + quad * 32 + lane;
#pragma unroll 1
        for (int cc = half * (BN / 32); cc < (half + 1) * (BN / 32); cc++) {
            unsigned r[16];
            const unsigned taddr = tmem + ((unsigned)(quad * 32) << 16) + (unsigned)(cc * 16);
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                           "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
                           "=r"(r[14]), "=r"(r[15])
                         : "r"(taddr));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            gemm_epilogue16(g, row, n0 + cc * 16, r);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((unsigned)BN));
}

static bool gemm_args_ok(const GemmArgs &a)
{
    const int am = a.a_t ? a.M : a.K, bm = a.b_t ? a.N : a.K;
    if (a.K % 8 || a.lda % 8 || a.ldb % 8 || a.lda < am || a.ldb < bm || ((uintptr_t)a.A & 15) ||
        ((uintptr_t)a.B & 15) || !a.err) {
        set_error(FDTD_ERR_ARG, "gemm: K %d, lda %d, ldb %d must be multiples of 8 (>= K), operands 16-byte aligned",
                  a.K, a.lda, a.ldb);
        return false;
    }
    return true;
}

template <int BN> static bool launch_group(GemmGroup &grp, bool two, bool sums, cudaStream_t st)
{
    int blocks = 0;
    for (int p = 0; p < 2; p++) {
        const GemmArgs &g = grp.g[p];
        grp.cols[p] = p == 0 || two ? (g.N + BN - 1) / BN : 1;
        grp.tiles[p] = p == 0 || two ? ((g.M + kGemmBM - 1) / kGemmBM) * grp.cols[p] : 0;
        blocks += grp.tiles[p];
    }
    if (sums) blocks += (grp.cs.cols + kSumCols - 1) / kSumCols;
    const int smem = kGemmStages * stage_bytes<BN>();
    // per device, and cheap: set on every launch
    if (!cuda_ok(cudaFuncSetAttribute(k_umma_gemm<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), "gemm smem"))
        return false;
    note_launch();
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cuda_ok(cudaLaunchKernelEx(&cfg, k_umma_gemm<BN>, grp), "gemm launch");
}

static long long tiles32(const GemmArgs &g)
{
    return (long long)((g.M + kGemmBM - 1) / kGemmBM) * ((g.N + 31) / 32);
}

bool gemm_bf16_group(const GemmArgs &g0, const GemmArgs *g1, const ColSum *cs, cudaStream_t st)
{
    if (!gemm_args_ok(g0) || (g1 && !gemm_args_ok(*g1))) return false;
    GemmGroup grp{};
    grp.g[0] = g0;
    if (g1) grp.g[1] = *g1;
    if (cs) grp.cs = *cs;
    const long long tiles = tiles32(g0) + (g1 ? tiles32(*g1) : 0);
    return tiles <= 2 * 148 ? launch_group<32>(grp, g1 != nullptr, cs != nullptr, st)
                            : launch_group<128>(grp, g1 != nullptr, cs != nullptr, st);
}

bool gemm_bf16_launch(const GemmArgs &a, cudaStream_t st)
{
    if (a.M <= 0 || a.N <= 0 || a.K <= 0) return true;
    return gemm_bf16_group(a, nullptr, nullptr, st);
}

}  // namespace fdtd

using namespace fdtd;

extern "C" int fdtd_gemm_bf16(const void *A, int lda, const void *B, int ldb, int M, int N, int K, const float *bias,
                              int act, float alpha, float beta, float *C32, int ldc32, void *C16, int ldc16,
                              float *Z32, int ldz, int *err, void *stream)
{
    if (!device_available()) return fdtd_last_error();
    if ((beta != 0.0f && !C32) || act < 0 || act > 1) {
        set_error(FDTD_ERR_ARG, "fdtd_gemm_bf16: beta needs C32; act must be 0 or 1");
        return FDTD_ERR_ARG;
    }
    GemmArgs a{(const __nv_bfloat16 *)A, (const __nv_bfloat16 *)B, lda, ldb, M, N, K, bias, act, alpha, beta,
               C32, ldc32, (__nv_bfloat16 *)C16, ldc16, Z32, ldz, err, false, false, nullptr};
    return gemm_bf16_launch(a, (cudaStream_t)stream) ? FDTD_OK : fdtd_last_error();
}
