// surrogate.cu -- the surrogate network of the taper optimiser: an MLP
// n_in -> H -> H -> H -> n_out with GELU (20 -> 256 -> 256 -> 256 -> 22 in the
// optimiser: 142,614 parameters), BF16 weights and activations, FP32
// accumulation on the tcgen05 tensor cores (umma_gemm.cu), FP32 master
// weights, Adam.  New work (the reference optimises by the adjoint gradient
// alone); its CPU FP64 restatement is oracle/surrogate.py.
//
// Layout: layer l maps in_l -> out_l; W_l is stored [out_l][in_pad_l] (FP32
// master and BF16 copy; the backward GEMM reads the copy transposed); padded
// columns are zero and stay zero (the padded inputs are zero, so their
// gradients are).
// Forward: Z_l = H_{l-1} W_l^T + b_l (FP32, kept), H_l = bf16(GELU(Z_l)),
// Y = H_3 W_4^T + b_4 (FP32).  Loss: mean over batch and outputs of (Y-T)^2.
// Backward per layer: db = column sums of dZ (FP32), dW = dZ^T H_{l-1}
// (GEMM over the batch, both operands read transposed), dH_{l-1} = dZ W_l,
// dZ_{l-1} = dH_{l-1} GELU'(Z_{l-1}) in its epilogue; dX = dZ_1 W_1 for the
// input gradient.  All of a layer's backward is one launch.  Rounding points (BF16 operands of every GEMM) are the ones
// the restatement reproduces.
#include <algorithm>
#include <cmath>
#include <cuda_bf16.h>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "engine.h"

namespace fdtd {

namespace {

constexpr int kLayers = 4;

int pad8(int x) { return (x + 7) / 8 * 8; }

// f32 [rows][cols] -> bf16 [rows][ldo] (columns cols..ldo-1 zero)
__global__ void k_pack_bf16(const float *in, int rows, int cols, int ldi, __nv_bfloat16 *out, int ldo)
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const long long n = (long long)rows * ldo;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(t / ldo), c = (int)(t % ldo);
        out[t] = __float2bfloat16_rn(c < cols ? in[(long long)r * ldi + c] : 0.0f);
    }
}

// dZ = 2 (Y - T) / (B n) (f32 [B][n] and bf16 [B][np]); loss += sum (Y-T)^2 / (B n)
__global__ void k_mse(const float *Y, const float *T, int B, int n, int np, float *dZ, __nv_bfloat16 *dZb,
                      double *loss)
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const long long cnt = (long long)B * np;
    const float s = 2.0f / ((float)B * (float)n);
    double acc = 0.0;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < cnt; t += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(t / np), c = (int)(t % np);
        float g = 0.0f;
        if (c < n) {
            const float d = Y[(long long)r * n + c] - T[(long long)r * n + c];
            acc += (double)d * d;
            g = s * d;
            dZ[(long long)r * n + c] = g;
        }
        dZb[t] = __float2bfloat16_rn(g);
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0 && acc != 0.0) atomicAdd(loss, acc / ((double)B * n));
}

// given dY directly: dZ (f32 [B][n]) and bf16 [B][np]
__global__ void k_seed_grad(const float *dy, int B, int n, int np, float *dZ, __nv_bfloat16 *dZb)
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const long long cnt = (long long)B * np;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < cnt; t += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(t / np), c = (int)(t % np);
        const float g = c < n ? dy[(long long)r * n + c] : 0.0f;
        if (c < n) dZ[(long long)r * n + c] = g;
        dZb[t] = __float2bfloat16_rn(g);
    }
}

// Adam on every parameter of the network and the BF16 copy of them, in one
// launch over the contiguous parameter buffers (n a multiple of 4; padding has
// zero gradients and stays zero)
__global__ void k_adam(float4 *p, const float4 *g, float4 *m, float4 *v, __nv_bfloat162 *pb, long long n4, float lr,
                       float b1, float b2, float eps, float c1, float c2)
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    auto upd = [&](float &pt, float gt, float &mt, float &vt) {
        mt = b1 * mt + (1.0f - b1) * gt;
        vt = b2 * vt + (1.0f - b2) * gt * gt;
        pt -= lr * (mt / c1) / (sqrtf(vt / c2) + eps);
    };
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n4; t += (long long)gridDim.x * blockDim.x) {
        float4 pt = p[t], mt = m[t], vt = v[t];
        const float4 gt = g[t];
        upd(pt.x, gt.x, mt.x, vt.x);
        upd(pt.y, gt.y, mt.y, vt.y);
        upd(pt.z, gt.z, mt.z, vt.z);
        upd(pt.w, gt.w, mt.w, vt.w);
        p[t] = pt;
        m[t] = mt;
        v[t] = vt;
        pb[2 * t] = __nv_bfloat162(__float2bfloat16_rn(pt.x), __float2bfloat16_rn(pt.y));
        pb[2 * t + 1] = __nv_bfloat162(__float2bfloat16_rn(pt.z), __float2bfloat16_rn(pt.w));
    }
}

// launch with a programmatic dependency on the preceding kernel of the stream:
// every kernel here waits for it (griddepcontrol.wait) before it touches memory
template <typename... P, typename... A>
bool launch_chained(void (*k)(P...), int blocks, cudaStream_t st, A... args)
{
    note_launch();
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cuda_ok(cudaLaunchKernelEx(&cfg, k, P(args)...), "surrogate launch");
}

int blocks_for(long long n) { return (int)std::min<long long>((n + 255) / 256, 2368); }

struct Mlp {
    int nin = 0, hid = 0, nout = 0;
    int in[kLayers], inp[kLayers], out[kLayers], outp[kLayers];
    // parameters, gradients, Adam moments and the BF16 copy: one buffer each,
    // layer after layer W [outp][inp] (rows out.. and columns in.. zero), then b [outp]
    float *P = nullptr, *G = nullptr, *Mo = nullptr, *Vo = nullptr;
    __nv_bfloat16 *Pb = nullptr;
    long long total = 0;                     // elements of each, a multiple of 8
    float *W[kLayers] = {}, *b[kLayers] = {}, *gW[kLayers] = {}, *gb[kLayers] = {};
    __nv_bfloat16 *Wb[kLayers] = {};
    int step = 0;
    int cap = 0;
    float *xs = nullptr, *ts = nullptr, *dys = nullptr;   // f32 staging [cap][nin], [cap][nout]
    __nv_bfloat16 *X = nullptr;
    __nv_bfloat16 *H[kLayers] = {};
    float *Z[kLayers] = {}, *Y = nullptr, *dX = nullptr;
    float *dZf[2] = {};                      // dZ of a layer, FP32 and BF16; layers alternate
    __nv_bfloat16 *dZb[2] = {};
    double *loss = nullptr;
    int *err = nullptr;
    cudaStream_t st = nullptr;
    std::vector<void *> allocs;

    template <typename T> bool alloc(T **p, size_t count)
    {
        void *v = nullptr;
        if (!cuda_ok(cudaMalloc(&v, count * sizeof(T) + 16), "cudaMalloc(mlp)")) return false;
        allocs.push_back(v);
        *p = (T *)v;
        return cuda_ok(cudaMemsetAsync(v, 0, count * sizeof(T) + 16, st), "cudaMemsetAsync(mlp)");
    }
    ~Mlp()
    {
        if (st) cudaStreamSynchronize(st);
        for (void *p : allocs) cudaFree(p);
        if (st) cudaStreamDestroy(st);
    }
    long long wcount(int l) const { return (long long)outp[l] * inp[l]; }
    // host image of a parameter buffer <-> flat order W1 [out][in], b1, ..., unpadded
    void flatten(const float *img, float *flat) const;
    void unflatten(const float *flat, float *img) const;
    long long params() const
    {
        long long n = 0;
        for (int l = 0; l < kLayers; l++) n += (long long)out[l] * in[l] + out[l];
        return n;
    }
};

void Mlp::flatten(const float *img, float *flat) const
{
    for (int l = 0; l < kLayers; l++) {
        const float *w = img + (W[l] - P), *bb = img + (b[l] - P);
        for (int o = 0; o < out[l]; o++, flat += in[l]) std::copy(w + (size_t)o * inp[l], w + (size_t)o * inp[l] + in[l], flat);
        flat = std::copy(bb, bb + out[l], flat);
    }
}

void Mlp::unflatten(const float *flat, float *img) const
{
    std::fill(img, img + total, 0.0f);
    for (int l = 0; l < kLayers; l++) {
        float *w = img + (W[l] - P);
        for (int o = 0; o < out[l]; o++, flat += in[l]) std::copy(flat, flat + in[l], w + (size_t)o * inp[l]);
        std::copy(flat, flat + out[l], img + (b[l] - P));
        flat += out[l];
    }
}

bool mlp_setup(Mlp &m, int nin, int hid, int nout, unsigned long long seed)
{
    m.nin = nin; m.hid = hid; m.nout = nout;
    const int ins[kLayers] = {nin, hid, hid, hid}, outs[kLayers] = {hid, hid, hid, nout};
    for (int l = 0; l < kLayers; l++) {
        m.in[l] = ins[l]; m.inp[l] = pad8(ins[l]); m.out[l] = outs[l]; m.outp[l] = pad8(outs[l]);
    }
    if (!cuda_ok(cudaStreamCreateWithFlags(&m.st, cudaStreamNonBlocking), "stream")) return false;
    if (!m.alloc(&m.loss, 2)) return false;
    m.err = (int *)(m.loss + 1);             // read back together
    for (int l = 0; l < kLayers; l++) m.total += m.wcount(l) + m.outp[l];
    if (!m.alloc(&m.P, m.total) || !m.alloc(&m.G, m.total) || !m.alloc(&m.Mo, m.total) || !m.alloc(&m.Vo, m.total) ||
        !m.alloc(&m.Pb, m.total))
        return false;
    long long at = 0;
    for (int l = 0; l < kLayers; l++) {
        m.W[l] = m.P + at; m.gW[l] = m.G + at; m.Wb[l] = m.Pb + at;
        at += m.wcount(l);
        m.b[l] = m.P + at; m.gb[l] = m.G + at;
        at += m.outp[l];
    }
    // PyTorch-Linear-like init: U(-1/sqrt(in), 1/sqrt(in)), seeded splitmix64
    unsigned long long s = seed;
    auto uni = [&s]() {
        s += 0x9E3779B97F4A7C15ull;
        unsigned long long z = s;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return (double)(z >> 11) * (1.0 / 9007199254740992.0);
    };
    std::vector<float> flat, img((size_t)m.total);
    for (int l = 0; l < kLayers; l++) {
        const double bound = 1.0 / std::sqrt((double)m.in[l]);
        for (int q = 0; q < m.out[l] * m.in[l] + m.out[l]; q++) flat.push_back((float)((2 * uni() - 1) * bound));
    }
    m.unflatten(flat.data(), img.data());
    if (!cuda_ok(cudaMemcpyAsync(m.P, img.data(), img.size() * sizeof(float), cudaMemcpyHostToDevice, m.st), "init") ||
        !cuda_ok(cudaStreamSynchronize(m.st), "init"))
        return false;
    return true;
}

bool refresh_bf16(Mlp &m)
{
    const int row = 8;
    return launch_chained(k_pack_bf16, blocks_for(m.total), m.st, m.P, (int)(m.total / row), row, row, m.Pb, row);
}

bool ensure_cap(Mlp &m, int B)
{
    if (B <= m.cap) return true;
    // buffers sized for B (old ones stay allocated until the network is freed)
    const int h = m.hid, mx = std::max(m.hid, m.outp[kLayers - 1]);
    if (!m.alloc(&m.xs, (size_t)B * m.nin) || !m.alloc(&m.ts, (size_t)B * m.nout) ||
        !m.alloc(&m.dys, (size_t)B * m.nout) || !m.alloc(&m.X, (size_t)B * m.inp[0]) ||
        !m.alloc(&m.Y, (size_t)B * m.nout) || !m.alloc(&m.dX, (size_t)B * m.inp[0]))
        return false;
    for (int p = 0; p < 2; p++)
        if (!m.alloc(&m.dZf[p], (size_t)B * mx) || !m.alloc(&m.dZb[p], (size_t)B * mx)) return false;
    for (int l = 1; l < kLayers; l++)
        if (!m.alloc(&m.H[l], (size_t)B * h) || !m.alloc(&m.Z[l], (size_t)B * h))
            return false;
    m.cap = B;
    return true;
}

GemmArgs gemm(const Mlp &m, const __nv_bfloat16 *A, int lda, const __nv_bfloat16 *Bm, int ldb, int M, int N, int K)
{
    GemmArgs g{};
    g.A = A; g.lda = lda; g.B = Bm; g.ldb = ldb; g.M = M; g.N = N; g.K = K;
    g.alpha = 1.0f; g.beta = 0.0f; g.err = m.err;
    return g;
}

bool forward(Mlp &m, int B)
{
    if (!launch_chained(k_pack_bf16, blocks_for((long long)B * m.inp[0]), m.st, m.xs, B, m.nin, m.nin, m.X, m.inp[0]))
        return false;
    const __nv_bfloat16 *hin = m.X;
    int ldin = m.inp[0];
    for (int l = 0; l < kLayers; l++) {
        GemmArgs g = gemm(m, hin, ldin, m.Wb[l], m.inp[l], B, m.out[l], m.inp[l]);
        g.bias = m.b[l];
        if (l < kLayers - 1) {
            g.act = 1;
            g.Z32 = m.Z[l + 1]; g.ldz = m.hid;
            g.C16 = m.H[l + 1]; g.ldc16 = m.hid;
            hin = m.H[l + 1];
            ldin = m.hid;
        } else {
            g.C32 = m.Y; g.ldc32 = m.nout;
        }
        if (!gemm_bf16_launch(g, m.st)) return false;
    }
    return true;
}

// backward from dZ of the last layer (already in dZf[1] / dZb[1]); weight
// grads when `weights`, dX when `input`.  Per layer one launch: dW = dZ^T H (both
// operands read transposed), db, and dZ of the layer below (dH times GELU' in
// the epilogue), which goes to the other buffer.
bool backward(Mlp &m, int B, bool weights, bool input)
{
    for (int l = kLayers - 1; l >= 0; l--) {
        const int o = m.out[l], op = m.outp[l], ld = (l == kLayers - 1) ? op : m.hid, p = l & 1;
        GemmArgs dw = gemm(m, m.dZb[p], ld, l == 0 ? m.X : m.H[l], m.inp[l], o, m.inp[l], B);
        dw.a_t = dw.b_t = true;
        dw.C32 = m.gW[l]; dw.ldc32 = m.inp[l];
        GemmArgs dh = gemm(m, m.dZb[p], ld, m.Wb[l], m.inp[l], B, m.inp[l], op);
        dh.b_t = true;
        if (l > 0) {
            dh.act = 2; dh.Zin = m.Z[l]; dh.ldz = m.hid;
            dh.C32 = m.dZf[1 - p]; dh.ldc32 = m.hid;
            dh.C16 = m.dZb[1 - p]; dh.ldc16 = m.hid;
        } else {
            dh.C32 = m.dX; dh.ldc32 = m.inp[0];
        }
        const bool down = l > 0 || input;
        const ColSum cs{m.dZf[p], B, o, o, m.gb[l]};
        if (weights) {
            if (!gemm_bf16_group(dw, down ? &dh : nullptr, &cs, m.st)) return false;
        } else if (down && !gemm_bf16_group(dh, nullptr, nullptr, m.st)) {
            return false;
        }
    }
    return true;
}

bool upload(Mlp &m, float *dst, const float *src, size_t count)
{
    return cuda_ok(cudaMemcpyAsync(dst, src, count * sizeof(float), cudaMemcpyHostToDevice, m.st), "mlp H2D");
}

// waits for the network's stream; the loss of the step when asked for
bool check_err(Mlp &m, double *loss = nullptr)
{
    struct { double loss; int err, pad; } r{};
    static_assert(sizeof r == 2 * sizeof(double), "status layout");
    if (!cuda_ok(cudaMemcpyAsync(&r, m.loss, sizeof r, cudaMemcpyDeviceToHost, m.st), "status D2H") ||
        !cuda_ok(cudaStreamSynchronize(m.st), "mlp sync"))
        return false;
    if (loss) *loss = r.loss;
    if (r.err) {
        cudaMemsetAsync(m.err, 0, sizeof(int), m.st);
        set_error(FDTD_ERR_TIMEOUT, "surrogate: a tensor-core GEMM wait gave up");
        return false;
    }
    return true;
}

bool batch_ok(const Mlp *m, int B)
{
    if (!m || B <= 0 || B % 8) {
        set_error(FDTD_ERR_ARG, "surrogate: batch %d must be a positive multiple of 8", B);
        return false;
    }
    return true;
}

std::vector<Mlp *> &nets()
{
    static std::vector<Mlp *> v;
    return v;
}

Mlp *net(void *h)
{
    for (auto *p : nets())
        if (p == h) return p;
    set_error(FDTD_ERR_ARG, "surrogate: unknown network handle");
    return nullptr;
}

}  // namespace
}  // namespace fdtd

using namespace fdtd;

extern "C" {

void *fdtd_mlp_new(int n_in, int hidden, int n_out, unsigned long long seed)
{
    std::lock_guard<std::mutex> lock(api_mutex());
    if (!device_available()) return nullptr;
    if (n_in <= 0 || hidden <= 0 || hidden % 8 || n_out <= 0) {
        set_error(FDTD_ERR_ARG, "fdtd_mlp_new: n_in %d hidden %d (multiple of 8) n_out %d", n_in, hidden, n_out);
        return nullptr;
    }
    auto *m = new Mlp;
    if (!mlp_setup(*m, n_in, hidden, n_out, seed) || !refresh_bf16(*m) || !check_err(*m)) {
        delete m;
        return nullptr;
    }
    nets().push_back(m);
    return m;
}

long long fdtd_mlp_param_count(void *h)
{
    std::lock_guard<std::mutex> lock(api_mutex());
    Mlp *m = net(h);
    return m ? m->params() : -1;
}

// flat order: W_1 [out][in], b_1, ..., W_4, b_4 (unpadded)
int fdtd_mlp_get_params(void *h, float *out)
{
    std::lock_guard<std::mutex> lock(api_mutex());
    Mlp *m = net(h);
    if (!m || !out) return FDTD_ERR_ARG;
    if (!cuda_ok(cudaStreamSynchronize(m->st), "sync")) return fdtd_last_error();
    std::vector<float> img((size_t)m->total);
    if (!cuda_ok(cudaMemcpy(img.data(), m->P, img.size() * sizeof(float), cudaMemcpyDeviceToHost), "D2H"))
        return fdtd_last_error();
    m->flatten(img.data(), out);
    return FDTD_OK;
}

int fdtd_mlp_set_params(void *h, const float *in)
{
    std::lock_guard<std::mutex> lock(api_mutex());
    Mlp *m = net(h);
    if (!m || !in) return FDTD_ERR_ARG;
    if (!cuda_ok(cudaStreamSynchronize(m->st), "sync")) return fdtd_last_error();
    std::vector<float> img((size_t)m->total);
    m->unflatten(in, img.data());
    const size_t bytes = img.size() * sizeof(float);
    if (!cuda_ok(cudaMemcpyAsync(m->P, img.data(), bytes, cudaMemcpyHostToDevice, m->st), "H2D") ||
        !cuda_ok(cudaMemsetAsync(m->Mo, 0, bytes, m->st), "memset") ||
        !cuda_ok(cudaMemsetAsync(m->Vo, 0, bytes, m->st), "memset"))
        return fdtd_last_error();
    m->step = 0;
    return refresh_bf16(*m) && check_err(*m) ? FDTD_OK : fdtd_last_error();
}

int fdtd_mlp_forward(void *h, const float *x, int batch, float *y)
{
    std::lock_guard<std::mutex> lock(api_mutex());
    Mlp *m = net(h);
    if (!batch_ok(m, batch) || !x || !y) return FDTD_ERR_ARG;
    if (!ensure_cap(*m, batch) || !upload(*m, m->xs, x, (size_t)batch * m->nin) || !forward(*m, batch)) return fdtd_last_error();
    if (!cuda_ok(cudaMemcpyAsync(y, m->Y, (size_t)batch * m->nout * 4, cudaMemcpyDeviceToHost, m->st), "D2H"))
        return fdtd_last_error();
    return check_err(*m) ? FDTD_OK : fdtd_last_error();
}

static int grads_common(Mlp *m, const float *x, const float *t, int batch)
{
    if (!ensure_cap(*m, batch) || !upload(*m, m->xs, x, (size_t)batch * m->nin) ||
        !upload(*m, m->ts, t, (size_t)batch * m->nout) || !forward(*m, batch))
        return fdtd_last_error();
    if (!cuda_ok(cudaMemsetAsync(m->loss, 0, sizeof(double), m->st), "memset")) return fdtd_last_error();
    const int L = kLayers - 1;
    if (!launch_chained(k_mse, blocks_for((long long)batch * m->outp[L]), m->st, m->Y, m->ts, batch, m->nout, m->outp[L],
                        m->dZf[1], m->dZb[1], m->loss))
        return fdtd_last_error();
    if (!backward(*m, batch, true, false)) return fdtd_last_error();
    return FDTD_OK;
}

int fdtd_mlp_gradients(void *h, const float *x, const float *t, int batch, float *grad, double *loss)
{
    std::lock_guard<std::mutex> lock(api_mutex());
    Mlp *m = net(h);
    if (!batch_ok(m, batch) || !x || !t) return FDTD_ERR_ARG;
    int r = grads_common(m, x, t, batch);
    if (r != FDTD_OK || !check_err(*m, loss)) return r != FDTD_OK ? r : fdtd_last_error();
    if (grad) {
        std::vector<float> img((size_t)m->total);
        if (!cuda_ok(cudaMemcpy(img.data(), m->G, img.size() * sizeof(float), cudaMemcpyDeviceToHost), "D2H"))
            return fdtd_last_error();
        m->flatten(img.data(), grad);
    }
    return FDTD_OK;
}

int fdtd_mlp_train_step(void *h, const float *x, const float *t, int batch, float lr, double *loss)
{
    std::lock_guard<std::mutex> lock(api_mutex());
    Mlp *m = net(h);
    if (!batch_ok(m, batch) || !x || !t || !(lr > 0)) return FDTD_ERR_ARG;
    int r = grads_common(m, x, t, batch);
    if (r != FDTD_OK) return r;
    m->step++;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float c1 = 1.0f - std::pow(b1, (float)m->step), c2 = 1.0f - std::pow(b2, (float)m->step);
    if (!launch_chained(k_adam, blocks_for(m->total / 4), m->st, (float4 *)m->P, (const float4 *)m->G, (float4 *)m->Mo,
                        (float4 *)m->Vo, (__nv_bfloat162 *)m->Pb, m->total / 4, lr, b1, b2, eps, c1, c2))
        return fdtd_last_error();
    return check_err(*m, loss) ? FDTD_OK : fdtd_last_error();
}

int fdtd_mlp_input_gradient(void *h, const float *x, const float *dy, int batch, float *dx)
{
    std::lock_guard<std::mutex> lock(api_mutex());
    Mlp *m = net(h);
    if (!batch_ok(m, batch) || !x || !dy || !dx) return FDTD_ERR_ARG;
    if (!ensure_cap(*m, batch) || !upload(*m, m->xs, x, (size_t)batch * m->nin) ||
        !upload(*m, m->dys, dy, (size_t)batch * m->nout) || !forward(*m, batch))
        return fdtd_last_error();
    const int L = kLayers - 1;
    if (!launch_chained(k_seed_grad, blocks_for((long long)batch * m->outp[L]), m->st, m->dys, batch, m->nout,
                        m->outp[L], m->dZf[1], m->dZb[1]))
        return fdtd_last_error();
    if (!backward(*m, batch, false, true)) return fdtd_last_error();
    std::vector<float> full((size_t)batch * m->inp[0]);
    if (!cuda_ok(cudaMemcpyAsync(full.data(), m->dX, full.size() * 4, cudaMemcpyDeviceToHost, m->st), "D2H") ||
        !check_err(*m))
        return fdtd_last_error();
    for (int r = 0; r < batch; r++)
        for (int c = 0; c < m->nin; c++) dx[(size_t)r * m->nin + c] = full[(size_t)r * m->inp[0] + c];
    return FDTD_OK;
}

void fdtd_mlp_free(void *h)
{
    std::lock_guard<std::mutex> lock(api_mutex());
    auto &v = nets();
    for (size_t i = 0; i < v.size(); i++)
        if (v[i] == h) {
            delete v[i];
            v.erase(v.begin() + i);
            return;
        }
}

}  // extern "C"
