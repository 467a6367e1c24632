// yee_tile.cu -- the one-pass FP32 Yee step for grids whose three E coefficients
// agree in every cell (what every rasteriser writes; checked when materials are
// uploaded).  The scheme of yee_stream.cu: a block walks its tile's planes upwards,
// planes arrive two ahead in a ring of three stages, E and H of a plane in one pass,
// one block barrier a plane, every array read once and the other field set written.
//
// What bounds it is DRAM: a step has to move 52 B a cell (six fields and the
// coefficient read, six fields written; 60 with three coefficients) and 32 B more
// for every slab a cell lies in.  What differs from yee_stream.cu:
//  - a plane's rows of an array are one TMA box, seven a plane by one thread.  The
//    copies by 16-byte cp.async took the threads' issue slots (200x160x400 without
//    CPML: 144 us with them, 92 without any copies), and one 1-D bulk copy a row
//    waits in the copy engine (36 ns each).
//  - a quad's thread keeps the old H and new E of the plane below in registers, so
//    shared memory carries neighbours only; planes with and without slab cells are
//    loops of their own, and the slab auxiliaries of the next plane are loaded
//    before this one is computed (200x160x400 with CPML: 178 to 166 us).
//  - a row longer than a tile is split, so wide grids still get bands of seven rows.
//  - all columns are cut at the same planes, in one or two waves of blocks: tiles
//    that run side by side read a shared halo row from DRAM once (kInStep below).
// Per step, before (three coefficients, cp.async) and now: 200x160x400 with CPML 189
// and 158 us (5.07 TB/s of algorithmic bytes), with PEC 144 and 115 us; 384x256x384
// CPML 792 and 405; 256x128x128 CPML 77 and 68; 96x80x64 CPML, conductivity 45 and
// 14 us.  Two blocks an SM (96 registers) spill with CPML and gave nothing without.
#include "tile_cells.cuh"
#include "plane_ops.cuh"

#include <algorithm>

namespace fdtd {

constexpr int kTileMaxThreads = 512;

// the units of a chain (StepChain), unit u by warp u / blocks of block u % blocks
__device__ __forceinline__ void chain_units(const StepChain &c, int nx, int ny)
{
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int nov = c.sums ? c.njobs * c.nparts * 8 : 0;
    for (int u = (threadIdx.x >> 5) * c.blocks + blockIdx.x; u < c.units; u += nw * c.blocks) {
        if (u < nov) {
            const int part = (u >> 3) % c.nparts;
            const OverlapJob jb = c.jobs[(u >> 3) / c.nparts];
            double sre, sim;
            overlap_thread_sum<float>(c.f, nx, ny, jb, (u & 7) * 32 + lane, 256, part, c.nparts, sre, sim);
            overlap_warp_reduce(sre, sim);
            if (lane == 0) c.sums[u] = make_double2(sre, sim);
        } else if (u < nov + c.src_units) {
            mode_source_cells(c.src, (long long)(u - nov) * 32 + lane, (long long)c.src_units * 32,
                              schedule_step(c.src, *c.step + c.s + 1));
        } else {
            int cell = (u - nov - c.src_units) * 32;
            for (int b = 0; b < c.nstores; b++) {
                const ChainStore &d = c.store[b];
                if (cell >= 0 && cell < d.ncell) {
                    const int t = d.t0 + d.dir * (int)(*c.step + c.s - 1), e = cell + lane;
                    if (t >= 0 && t < d.duration && e < d.ncell) {
                        const long long q = d.cells[e];
                        float *dst = d.store + ((long long)t * d.ncell + e) * 3;
#pragma unroll
                        for (int m = 0; m < 3; m++) dst[m] = c.f[m][q];
                    }
                }
                cell -= (d.ncell + 31) / 32 * 32;
            }
        }
    }
}

template <bool CPML, bool LOSSY>
__global__ void __launch_bounds__(kTileMaxThreads, 1)
k_yee_tile(const __grid_constant__ StreamArgs a, const TileMaps *maps, const TileBox *tiles, TileShape sh,
           const __grid_constant__ StepChain chain, int *err)
{
    extern __shared__ __align__(128) float sm[];
    __shared__ TileSync sync;
    // programmatic dependent launch, as the other step kernels
    auto after_previous = []() {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    };
    if ((int)blockIdx.x == chain.ntiles) {
        after_previous();
        chain_add_up(chain.jobs, chain.njobs, chain.nparts, chain.prev, chain.scale, chain.dt, *chain.step + chain.s - 2,
                     threadIdx.x >> 5, blockDim.x >> 5);
        return;
    }
    tile_sync_init(&sync);
    // the descriptors, while the previous launch ends (0.3 us of a step)
    if (threadIdx.x < sizeof(TileMaps) / sizeof(CUtensorMap))
        asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<const CUtensorMap *>(maps) + threadIdx.x) : "memory");
    yee_tile<CPML, LOSSY>(a, maps, tiles[blockIdx.x], sh, sm, &sync, err, after_previous,
                          [&]() { if ((int)blockIdx.x < chain.blocks) chain_units(chain, a.nx, a.ny); });
}

using TileKernel = void (*)(StreamArgs, const TileMaps *, const TileBox *, TileShape, StepChain, int *);

static TileKernel tile_kernel(bool cpml, bool lossy)
{
    if (cpml) return lossy ? k_yee_tile<true, true> : k_yee_tile<true, false>;
    return lossy ? k_yee_tile<false, true> : k_yee_tile<false, false>;
}

// ---------------------------------------------------------------------------
// host side: the tile plan
// ---------------------------------------------------------------------------
namespace {

struct Columns {
    std::vector<int> q;   // x tiles [q[c], q[c + 1])
    int tp = 0, sw = 0, threads = 0;
    size_t smem = 0;
};

// a row split into nxt tiles of about equal threads (a slab quad has four), the
// right halo quad of each but the last outside the x slabs; rows as many as fit
bool columns_of(int nx, int L, bool lossy, int nxt, Columns *out)
{
    const int QX = nx / 4;
    int QL = 0, QR = QX;
    if (L > 0) {
        QL = (L + 3) / 4;
        QR = std::min(std::max((nx - L) / 4, QL), QX);
    }
    if (nxt > 1 && (QR - QL) < 2 * nxt) return false;
    auto weight = [&](int q) { return q < QL || q >= QR ? 4 : 1; };
    int total = 0;
    for (int q = 0; q < QX; q++) total += weight(q);
    out->q.assign(1, 0);
    int acc = 0;
    for (int q = 0, c = 1; q < QX && c < nxt; q++) {
        if (acc * nxt >= total * c && q > QL && q < QR && q > out->q.back()) {
            out->q.push_back(q);
            c++;
        }
        acc += weight(q);
    }
    if ((int)out->q.size() != nxt) return false;
    out->q.push_back(QX);
    out->sw = 0;   // a halo quad at every cut
    for (int c = 0; c < nxt; c++) out->sw = std::max(out->sw, out->q[c + 1] - out->q[c] + (c > 0) + (c + 1 < nxt));
    out->tp = 0;
    for (int tp = 2; tp <= 65; tp++) {
        int th = 0;
        for (int c = 0; c < nxt; c++) th = std::max(th, tile_roles(nx, L, out->q[c], out->q[c + 1], tp).threads);
        const TileShape sh{tp, out->sw};
        const size_t bytes = sh.floats(lossy, L) * sizeof(float);
        if (th > kTileMaxThreads || !sh.fits(lossy) || bytes > kStreamSmemBudget) break;
        out->tp = tp;
        out->threads = th;
        out->smem = bytes;
    }
    return out->tp >= 2;
}

// Time of a plane's pass of a tile of `quads` x `rows` (us; only ratios matter),
// from timing every tile of a 200x160x400 and a 256x128x128 grid: bands of 5 and 6
// rows outside the y slabs 1.53 and 1.65 us (64 quads: 4 and 5 rows 1.62 and 1.77),
// in them 3.12 and 3.15 (3 and 4 rows 2.90 and 2.97); a z-slab plane is 1.8 to 1.95
// planes.  A tile also makes the E pass of the plane above it, and starts.
double plane_cost(bool y_slab, int quads, int rows)
{
    const double w = quads / 50.0;
    return y_slab ? 2.60 + 0.09 * w * rows : 0.90 + 0.13 * w * rows;
}
double plane_weight(int nz, int L, int k) { return L > 0 && (k < L || k >= nz - L) ? 1.9 : 1.0; }
constexpr double kTileStart = 1.5;

// Cuts at the same planes keep neighbouring tiles in step, so that a halo row is
// read from DRAM by one of them only: 200x160x400 without CPML moves 622 MB a step
// against 705, in 123 us against 138.
constexpr double kInStep = 0.88;

// the rows 1..ny-2 between the y-slab edges; above the interior the cut is one row
// early, so that no interior band's halo row lies in the slab
struct Segment { int row, len; bool y_slab; };
std::vector<Segment> segments(int ny, int L)
{
    std::vector<Segment> out;
    for (int t0 = 0; t0 < ny - 2;) {
        int t1 = t0 + 1;
        while (t1 < ny - 2 && !(L > 0 && (1 + t1 == L || 1 + t1 == ny - L - 1))) t1++;
        out.push_back(Segment{1 + t0, t1 - t0, L > 0 && (1 + t0 < L || t1 >= ny - L)});
        t0 = t1;
    }
    return out;
}

// the columns (bands of rows x ranges of quads) a grid is cut into
struct ColumnSet {
    int tp = 0, threads = 0;
    std::vector<TileBox> box;            // planes 1..nz-2 each
    std::vector<double> plane;           // a plane's pass
    std::vector<char> y_slab;
    int bands[2] = {0, 0};               // columns outside and inside the y slabs
    double most[2] = {0, 0};             // the largest pass of each kind
};

// bands of at most cap[in y slabs] rows, of even size between the y-slab edges
void cut_bands(const std::vector<Segment> &seg, int nx, int nz, int L, const Columns &col, const int cap[2], ColumnSet *out)
{
    const int nxt = (int)col.q.size() - 1;
    int most = 0;
    *out = ColumnSet{};
    for (const Segment &s : seg) {
        const int parts = (s.len + cap[s.y_slab] - 1) / cap[s.y_slab];
        for (int p = 0; p < parts; p++) {
            const int r0 = (int)((long long)s.len * p / parts), r1 = (int)((long long)s.len * (p + 1) / parts);
            most = std::max(most, r1 - r0);
            for (int c = 0; c < nxt; c++) {
                const double t = plane_cost(s.y_slab, col.q[c + 1] - col.q[c], r1 - r0);
                out->box.push_back(TileBox{col.q[c], col.q[c + 1], s.row + r0, r1 - r0, 1, nz - 1});
                out->plane.push_back(t);
                out->y_slab.push_back(s.y_slab);
                out->bands[s.y_slab]++;
                out->most[s.y_slab] = std::max(out->most[s.y_slab], t);
            }
        }
    }
    out->tp = most + 1;
    for (int c = 0; c < nxt; c++)
        out->threads = std::max(out->threads, tile_roles(nx, L, col.q[c], col.q[c + 1], out->tp).threads);
}

// The columns laid end to end and cut into shares of `span`: a share is one tile,
// or the end of a column and the start of the next (no tile shorter than 4 planes).
// Returns the number of shares; the tiles' costs with them.
int deal(const ColumnSet &c, const std::vector<double> &weight, double span, std::vector<TileBox> *tiles,
         std::vector<double> *cost)
{
    const int planes = (int)weight.size();
    int shares = 0;
    double left = 0;
    for (size_t b = 0; b < c.box.size(); b++) {
        for (int p = 0; p < planes;) {
            const double unit = c.plane[b];
            // a new share when what is left holds no tile worth its start
            if (left < kTileStart + unit * (1 + 4 * weight[p])) {
                shares++;
                left = span;
            }
            double acc = kTileStart + unit;
            int q = p;
            while (q < planes && (q - p < 4 || planes - q < 4 || acc + unit * weight[q] <= left)) acc += unit * weight[q++];
            if (q < planes)
                while (planes - q < 4 && q - p > 4) acc -= unit * weight[--q];
            if (tiles) {
                TileBox t = c.box[b];
                t.k0 = 1 + p;
                t.k1 = 1 + q;
                tiles->push_back(t);
                cost->push_back(acc);
            }
            left -= acc;
            p = q;
        }
    }
    return shares;
}

// Shares for nsm blocks, the longest tiles first: the hardware starts blocks in
// order as others end, so a share's short rest lands behind about the tile that it
// was cut from.
double plan_shares(const ColumnSet &c, const std::vector<double> &weight, int nsm, std::vector<TileBox> *out)
{
    double w = 0, hi = 0;
    for (double x : weight) w += x;
    for (double p : c.plane) hi += p * (w + 1) + kTileStart;
    double lo = hi / nsm * 0.5;
    for (int i = 0; i < 30; i++) {
        const double mid = 0.5 * (lo + hi);
        (deal(c, weight, mid, nullptr, nullptr) <= nsm ? hi : lo) = mid;
    }
    std::vector<TileBox> tiles;
    std::vector<double> cost;
    deal(c, weight, hi, &tiles, &cost);
    std::vector<int> order(tiles.size());
    for (size_t i = 0; i < order.size(); i++) order[i] = (int)i;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return cost[x] > cost[y]; });
    std::vector<double> busy(nsm, 0.0);
    out->clear();
    for (int i : order) {
        out->push_back(tiles[i]);
        *std::min_element(busy.begin(), busy.end()) += cost[i];
    }
    return *std::max_element(busy.begin(), busy.end());
}

// n[0] chunks of planes of every column outside the y slabs, n[1] of those inside:
// the time of the launch when there are at most 2 nsm tiles, the longer first
double chunk_span(const ColumnSet &c, double w, const int n[2], int nsm)
{
    double t[2];
    int cnt[2];
    for (int y = 0; y < 2; y++) {
        cnt[y] = c.bands[y] * n[y];
        t[y] = cnt[y] ? kTileStart + c.most[y] * (w / n[y] + 1) : 0;
    }
    const int hi = t[1] > t[0];
    const double a = t[hi], b = t[1 - hi];
    const int rest = cnt[0] + cnt[1] - nsm;   // tiles of the second wave
    if (rest <= 0) return a;
    if (cnt[hi] > nsm) return 2 * a;
    return rest <= nsm - cnt[hi] ? std::max(a, 2 * b) : a + b;
}

// those tiles: all columns' first chunks, then the second, ... of the longer kind first
void plan_chunks(const ColumnSet &c, const std::vector<double> &weight, double w, const int n[2], std::vector<TileBox> *out)
{
    const int planes = (int)weight.size();
    auto cuts = [&](int m) {
        std::vector<int> at(1, 0);
        double acc = 0;
        for (int q = 0; q < planes; q++) {
            acc += weight[q];
            // chunk i ends here; where as many planes are left as chunks, each is one
            // (a cut that was let pass there left all the rest to one chunk: 48x40x44
            // with a 6-cell CPML had a tile of 19 planes and took 44.6 us, now 9.7)
            const int i = (int)at.size(), spare = planes - q - 1 - (m - i);
            if (i < m && spare >= 0 && (spare == 0 || acc >= w * i / m - 0.5 * weight[q])) at.push_back(q + 1);
        }
        at.push_back(planes);
        return at;
    };
    const int first = c.most[1] * (w / n[1] + 1) > c.most[0] * (w / n[0] + 1);
    out->clear();
    for (int y : {first, 1 - first}) {
        const std::vector<int> at = cuts(n[y]);
        for (size_t i = 0; i + 1 < at.size(); i++)
            for (size_t b = 0; b < c.box.size(); b++) {
                if (c.y_slab[b] != y) continue;
                TileBox t = c.box[b];
                t.k0 = 1 + at[i];
                t.k1 = 1 + at[i + 1];
                out->push_back(t);
            }
    }
}

}  // namespace

// rows in as few tiles as fit: a second tile a row costs more than the wider bands
// save (200 cells without CPML, in halves: 159 us against 123), since its edges split
// lines and DRAM bursts
static bool tile_columns(int nx, int L, bool lossy, Columns *col)
{
    for (int nxt = 1; nxt <= 8; nxt++)
        if (columns_of(nx, L, lossy, nxt, col)) return true;
    return false;
}

int tile_supported(int nx, int ny, int nz, bool lossy, int L)
{
    if (nx % 4 != 0 || nx < 8 || ny < 3 || nz < 3 || L < 0) return 0;
    if ((long long)nx * ny * nz >= (1LL << 31)) return 0;   // cell indices are 32-bit (sidx_t)
    Columns c;
    return tile_columns(nx, L, lossy, &c);
}

bool tile_plan(int nx, int ny, int nz, int L, bool lossy, int nsm, TilePlan *out)
{
    if (!tile_supported(nx, ny, nz, lossy, L) || nsm <= 0) return false;
    Columns col;
    if (!tile_columns(nx, L, lossy, &col)) return false;
    std::vector<double> weight;
    double w = 0;
    for (int k = 1; k <= nz - 2; k++) {
        weight.push_back(plane_weight(nz, L, k));
        w += weight.back();
    }
    const std::vector<Segment> seg = segments(ny, L);
    const int most = col.tp - 1;
    ColumnSet c, best;
    int cap[2] = {most, most}, n[2], best_n[2] = {0, 0};
    cut_bands(seg, nx, nz, L, col, cap, &c);
    out->tiles.clear();
    out->span = plan_shares(c, weight, nsm, &out->tiles);
    best = c;
    // bands of half the rows at least, one or two waves of tiles
    int seen[2] = {0, 0};
    for (cap[0] = most; 2 * cap[0] >= most; cap[0]--) {
        for (cap[1] = most; 2 * cap[1] >= most; cap[1]--) {
            cut_bands(seg, nx, nz, L, col, cap, &c);
            if (c.bands[0] == seen[0] && c.bands[1] == seen[1]) continue;
            seen[0] = c.bands[0];
            seen[1] = c.bands[1];
            for (int waves = 1; waves <= 2; waves++)
                for (n[0] = 1; n[0] <= nz - 2; n[0]++) {
                    const int room = waves * nsm - n[0] * c.bands[0];
                    if (room < c.bands[1]) break;
                    n[1] = c.bands[1] ? std::min(room / c.bands[1], nz - 2) : 1;
                    if (c.bands[0] == 0 && n[0] > 1) break;
                    const double t = kInStep * chunk_span(c, w, n, nsm);
                    if (t >= out->span) continue;
                    out->span = t;
                    best = c;
                    best_n[0] = n[0];
                    best_n[1] = n[1];
                }
            if (c.bands[1] == 0) break;
        }
    }
    if (best_n[0]) plan_chunks(best, weight, w, best_n, &out->tiles);
    out->tp = best.tp;
    out->sw = col.sw;
    out->threads = best.threads;
    out->smem = TileShape{out->tp, out->sw}.floats(lossy, L) * sizeof(float);
    return true;
}

// (the limit is the kernel's, not a grid's: always the same one, so that no plan takes
// it from the grids prepared before; a launch names its own size)
bool tile_configure(size_t smem, int threads)
{
    if (smem > kStreamSmemBudget) return false;
    for (int v = 0; v < 4; v++) {
        const void *f = (const void *)tile_kernel((v & 2) != 0, (v & 1) != 0);
        cudaFuncAttributes at{};
        if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStreamSmemBudget) != cudaSuccess ||
            cudaFuncGetAttributes(&at, f) != cudaSuccess || at.maxThreadsPerBlock < threads)
            return false;
    }
    return true;
}

bool tile_make_maps(TileMaps *m, const float *const f[6], const float *cb, const float *ca, int nx, int ny, int nz,
                    const TilePlan &p)
{
    const int bx = 4 * p.sw;
    for (int c = 0; c < 3; c++)
        if (!tma_encode_3d(&m->h[c], f[3 + c], nx, ny, nz, bx, p.tp + 1) ||
            !tma_encode_3d(&m->e[c], f[c], nx, ny, nz, bx, p.tp))
            return false;
    return tma_encode_3d(&m->cb, cb, nx, ny, nz, bx, p.tp) && tma_encode_3d(&m->ca, ca ? ca : cb, nx, ny, nz, bx, p.tp);
}

void launch_yee_tile(const StreamArgs &a, const TileMaps *maps, const TileBox *tiles, const TilePlan &p, StepChain chain,
                     int *err, cudaStream_t st)
{
    note_launch(1);
    chain.ntiles = (int)p.tiles.size();
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(chain.ntiles + (chain.prev ? 1 : 0)));
    cfg.blockDim = dim3((unsigned)p.threads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, tile_kernel(a.L > 0, a.ca[0] != nullptr), a, maps, tiles, TileShape{p.tp, p.sw}, chain, err);
}

// a plane's wait for a copy that never comes (fdtd_wait_selftest): gives up, and the
// next wait sees that at once
__global__ void k_tile_wait_selftest(unsigned long long limit_ns, int *err, unsigned long long *elapsed_ns)
{
    __shared__ TileSync sync;
    tile_sync_init(&sync);
    __syncthreads();
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    const bool landed = tile_wait(&sync, &sync.full[0], 0, false, limit_ns);
    __syncthreads();
    const bool later = tile_wait(&sync, &sync.full[1], 0, false, limit_ns);
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
    if (threadIdx.x != 0) return;
    if (!landed && !later && *(volatile int *)&sync.abort) atomicExch(err, 1);
    *elapsed_ns = t1 - t0;
}

void launch_tile_wait_selftest(unsigned long long limit_ns, int *err, unsigned long long *elapsed_ns, cudaStream_t st)
{
    note_launch();
    k_tile_wait_selftest<<<1, 32, 0, st>>>(limit_ns, err, elapsed_ns);
}

}  // namespace fdtd

// ---------------------------------------------------------------------------
// plan inspection (host only; no device work)
// ---------------------------------------------------------------------------
extern "C" int fdtd_tile_plan(int nx, int ny, int nz, int cpml_cells, int lossy, int nsm, int *tiles, int cap,
                              int *staged_rows, int *threads, long long *smem_bytes)
{
    using namespace fdtd;
    if (cpml_cells < 0 || nsm <= 0 || !staged_rows || !threads || !smem_bytes) return -1;
    TilePlan p;
    if (!tile_plan(nx, ny, nz, cpml_cells, lossy != 0, nsm, &p)) return -1;
    *staged_rows = p.tp;
    *threads = p.threads;
    *smem_bytes = (long long)p.smem;
    if (tiles) {
        if (cap < (int)p.tiles.size()) return -1;
        for (const TileBox &t : p.tiles) {
            const int v[6] = {t.q0, t.q1, t.j0, t.rows, t.k0, t.k1};
            tiles = std::copy(v, v + 6, tiles);
        }
    }
    return (int)p.tiles.size();
}
