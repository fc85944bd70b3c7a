// C ABI of the B200 extrapolation + imaging library: plans, kernel dispatch and the
// reference-compatible entry points.  Declarations and contracts: include/imaging2d_wlsq_b200.h.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <condition_variable>
#include <map>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <mutex>
#include <numeric>
#include <string>
#include <thread>
#include <vector>

#include "../../include/imaging2d_wlsq_b200.h"
#include <cufft.h>
#include "wlsq_kernels.cuh"
#include "wlsq_cluster.cuh"
#include "wlsq_cluster2.cuh"
#include "wlsq_rows.cuh"
#include "wlsq_wide.cuh"
#include "wlsq_adjoint.cuh"
#include "wlsq_adjoint_cluster.cuh"
#include "wlsq_rows_adjoint.cuh"
#include "wlsq_adjoint_wide.cuh"
#include "wlsq_frontend.cuh"

namespace img2d {

static thread_local std::string g_err;

static int fail(int code, const std::string &msg)
{
    g_err = msg;
    return code;
}

#define IMG2D_CUDA(call)                                                                   \
    do {                                                                                   \
        cudaError_t e_ = (call);                                                           \
        if (e_ != cudaSuccess) {                                                           \
            cudaGetLastError();                                                            \
            return fail(e_ == cudaErrorMemoryAllocation ? IMG2D_ENOMEM : IMG2D_ECUDA,      \
                        std::string(#call) + ": " + cudaGetErrorString(e_));               \
        }                                                                                  \
    } while (0)

typedef void (*KernelFn)(MigrateArgs);

// ---------------------------------------------------------------------------------------
// Kernel tables.  The fixed-length kernel is instantiated for the operator lengths of the
// reference tests and of the benchmark configurations; any other length runs on the generic
// kernel.
// ---------------------------------------------------------------------------------------
constexpr int kX = 8;

template <int G, int L>
struct FixedEntry {
    static constexpr int g = G, l = L;
};

struct FixedKernel {
    int G, L;
    KernelFn fn;
};

#define IMG2D_FIXED(G, L) {G, L, migrate_fixed_kernel<G, kX, L, OP_CONJ>}
#define IMG2D_FIXED_L(L) IMG2D_FIXED(1, L), IMG2D_FIXED(2, L), IMG2D_FIXED(4, L), IMG2D_FIXED(8, L)

static const FixedKernel kFixed[] = {
    IMG2D_FIXED_L(3),  IMG2D_FIXED_L(5),  IMG2D_FIXED_L(11), IMG2D_FIXED_L(25),
    IMG2D_FIXED_L(31), IMG2D_FIXED_L(35), IMG2D_FIXED_L(43), IMG2D_FIXED_L(55),
};

static KernelFn find_fixed(int G, int L)
{
    for (const auto &k : kFixed)
        if (k.G == G && k.L == L) return k.fn;
    return nullptr;
}

// Row-split kernels by slots per item, tap pairs per lane and number of tables; 4 outputs per quad, a
// row's next taps held in registers.  Tried on one shot of 1024 x 500, 256 frequencies, 31 taps (3.36
// ms) and slower: 8 outputs per quad (3.58 ms, 168 registers; 3.45 without the held taps), three CTAs
// per SM at 80 registers (3.76), 4 slots per item (spills).  With two slots packed multiply-adds and
// held taps together gave 3 to 6% (9 shots, two tables: 643 -> 603 us), neither alone did.
struct RowsKernel {
    int G, np;
    bool two;
    KernelFn fn;
};
#define IMG2D_ROWS(NP)                                                                         \
    {1, NP, false, migrate_rows_kernel<1, NP, false>}, {1, NP, true, migrate_rows_kernel<1, NP, true>},  \
        {2, NP, false, migrate_rows_kernel<2, NP, false>}, {2, NP, true, migrate_rows_kernel<2, NP, true>}
static const RowsKernel kRows[] = {
    IMG2D_ROWS(1), IMG2D_ROWS(2), IMG2D_ROWS(3), IMG2D_ROWS(4), IMG2D_ROWS(5),
    IMG2D_ROWS(6), IMG2D_ROWS(7), IMG2D_ROWS(8), IMG2D_ROWS(10),
};

static KernelFn find_rows(int G, int L, bool two)
{
    if (L < 3) return nullptr;
    for (const auto &k : kRows)
        if (k.G == G && k.np == rows_np(L) && k.two == two) return k.fn;
    return nullptr;
}

// Threads per CTA and estimated time of the row-split kernel, in microseconds per depth step, for
// n_items items of windows up to W.  A step of a CTA is `rounds` blocks per warp, each taking
// 0.45 us (1 + k / 6) with k warps on the SM, times 1.45 for two slots (fitted on a B200, 31 taps,
// one table: 3 to 16 warps per SM; within 15% on the cases it was checked on); items beyond what is
// resident run in further waves.  At most `most` CTAs share an SM.
struct RowsLaunch {
    int warps;
    double us;
};
static RowsLaunch rows_launch(int G, int W, int L, bool two, long long n_items, int nsm, size_t smem_sm, int most)
{
    const int nwb = (W + kRowsWarpPos - 1) / kRowsWarpPos;
    const size_t smem = rows_smem_bytes(G, W, L) + 1024;
    RowsLaunch best{1, 1e30};
    for (int w = 1; w <= std::min(nwb, kRowsThreads / 32); ++w) {
        const long long c = std::min<long long>({16 / w, (long long)(smem_sm / smem), most});  // 128 registers a thread
        if (c < 1) continue;
        const int rounds = (nwb + w - 1) / w;
        auto wave = [&](long long per_sm) { return rounds * 0.45 * (1.0 + per_sm * w / 6.0); };
        const long long full = n_items / (nsm * c), rest = n_items % (nsm * c);
        double us = full * wave(c) + (rest ? wave((rest + nsm - 1) / nsm) : 0.0);
        us *= (G == 2 ? 1.45 : 1.0) * (two ? 1.2 : 1.0) * (0.25 + 0.75 * rows_np(L) / 4);
        if (us < best.us) best = RowsLaunch{w, us};
    }
    return best;
}

// Time at which the last of nf items of each cost is done, taken in order of falling cost by `workers`.
static double queue_time(std::vector<double> cost, int nf, int workers)
{
    std::sort(cost.begin(), cost.end(), std::greater<double>());
    const double sum = std::accumulate(cost.begin(), cost.end(), 0.0) * nf;
    const long long n = (long long)cost.size() * nf;
    if (n <= workers) return cost[0];
    // (many rounds: the last workers finish about half an item apart; stepping through 38000 items took 4 ms)
    if (n > 12ll * workers) return sum / workers + 0.5 * cost.back();
    std::vector<double> heap(workers, 0.0);  // when each worker is free, the earliest first
    for (double c : cost)
        for (int j = 0; j < nf; ++j) {
            std::pop_heap(heap.begin(), heap.end(), std::greater<double>());
            heap.back() += c;
            std::push_heap(heap.begin(), heap.end(), std::greater<double>());
        }
    return *std::max_element(heap.begin(), heap.end());
}

static KernelFn find_generic(int G, int mode)
{
#define IMG2D_GEN(GG)                                                        \
    if (G == GG) {                                                           \
        if (mode == OP_CONJ) return migrate_generic_kernel<GG, OP_CONJ>;     \
        if (mode == OP_TWO) return migrate_generic_kernel<GG, OP_TWO>;       \
        return migrate_generic_kernel<GG, OP_DENSE>;                         \
    }
    IMG2D_GEN(1) IMG2D_GEN(2) IMG2D_GEN(4) IMG2D_GEN(8)
#undef IMG2D_GEN
    return nullptr;
}

struct ClusterKernel {
    int L;
    KernelFn fn;
    size_t smem;
};

static const ClusterKernel kCluster[] = {
    {25, migrate_cluster_kernel<25>, cluster_smem_bytes<25>()},
    {31, migrate_cluster_kernel<31>, cluster_smem_bytes<31>()},
    {35, migrate_cluster_kernel<35>, cluster_smem_bytes<35>()},
    {43, migrate_cluster_kernel<43>, cluster_smem_bytes<43>()},
    {55, migrate_cluster_kernel<55>, cluster_smem_bytes<55>()},
};

// Variants of the second-generation cluster kernel: warps per CTA (positions per CTA = 32 * warps),
// operator-pair prefetch into registers, next-step operator rows prefetched into L1.
struct Cluster2Variant {
    int nw;
    bool tap_pf, row_pf;
    KernelFn fn;
    bool stage = false;  // uses the step-ahead shared-memory stage (cluster2_stage_bytes)
    bool ring = false;   // reads operator taps from the per-lane-group ring (cluster2_ring_bytes)
};

static const Cluster2Variant kCluster2[] = {
    {16, false, false, migrate_cluster2_kernel<16, false, false>},
    {16, false, true, migrate_cluster2_kernel<16, false, true>},
    {12, true, false, migrate_cluster2_kernel<12, true, false>},
    {12, true, true, migrate_cluster2_kernel<12, true, true>},
    {8, true, false, migrate_cluster2_kernel<8, true, false>},
    {8, true, true, migrate_cluster2_kernel<8, true, true>},
    {16, false, false, migrate_cluster2_kernel<16, false, false, true>},  // packed FFMA2 arithmetic
    {16, false, false, migrate_cluster2_kernel<16, false, false, false, TAB_F32, 1>},  // grouped FMA order
    {16, false, false, migrate_cluster2_kernel<16, false, false, false, TAB_F32, 2>},  // index prefetch
    {16, false, false, migrate_cluster2_kernel<16, false, false, false, TAB_F32, 3>},  // both
    {16, false, false, migrate_cluster2_kernel<16, false, false, false, TAB_F32, 4>, true},  // step-ahead stage
    {16, false, false, migrate_cluster2_kernel<16, false, false, false, TAB_F32, 8>, false, true},  // tap-pair ring
};
constexpr int kCluster2Staged = 10;   // 16 warps with the step-ahead shared-memory stage
constexpr int kCluster2Default = 11;  // 16 warps, tap pairs through the shared-memory ring
constexpr int kNumCluster2 = (int)(sizeof(kCluster2) / sizeof(kCluster2[0]));

// Demigration kernels: G lane slots per item, compile-time operator length (0 = runtime length).
constexpr int kAdjWarps = 16;
typedef void (*DemigFn)(DemigrateArgs);
struct DemigKernel {
    int G, L;
    DemigFn fn;
};
#define IMG2D_DEMIG(G, L) {G, L, demigrate_kernel<G, L, kAdjWarps>}
#define IMG2D_DEMIG_G(G) IMG2D_DEMIG(G, 0), IMG2D_DEMIG(G, 25), IMG2D_DEMIG(G, 31), IMG2D_DEMIG(G, 35), IMG2D_DEMIG(G, 55)
static const DemigKernel kDemig[] = {IMG2D_DEMIG_G(2), IMG2D_DEMIG_G(4), IMG2D_DEMIG_G(8)};

// Cluster demigration with unrolled steps.
static DemigFn find_demig_cluster(int L)
{
    return L == 25 ? demigrate_cluster_kernel<25> : (L == 31 ? demigrate_cluster_kernel<31> : (L == 35 ? demigrate_cluster_kernel<35> : nullptr));
}

// Row-split demigration kernels by slots per item and tap pairs per lane.
struct DemigRowsKernel {
    int NS, np;
    void (*fn)(RowsAdjArgs);
};
#define IMG2D_DROWS(NP) {1, NP, demigrate_rows_kernel<1, NP>}, {2, NP, demigrate_rows_kernel<2, NP>}
static const DemigRowsKernel kDemigRows[] = {
    IMG2D_DROWS(1), IMG2D_DROWS(2), IMG2D_DROWS(3), IMG2D_DROWS(4), IMG2D_DROWS(5),
    IMG2D_DROWS(6), IMG2D_DROWS(7), IMG2D_DROWS(8), IMG2D_DROWS(10),
};

static void (*find_demig_rows(int NS, int L))(RowsAdjArgs)
{
    if (L < 3) return nullptr;
    for (const auto &k : kDemigRows)
        if (k.NS == NS && k.np == rows_np(L)) return k.fn;
    return nullptr;
}

static DemigFn find_demig(int G, int L)
{
    DemigFn generic = nullptr;
    for (const auto &k : kDemig) {
        if (k.G != G) continue;
        if (k.L == L) return k.fn;
        if (k.L == 0) generic = k.fn;
    }
    return generic;
}

// Shared memory of the demigration kernel: one complex wavefield per slot, ping-pong.
static size_t demig_smem_bytes(int G, int W, int M)
{
    const int X = 8;
    const int Mp = ((M + X - 1) / X) * X;
    const int Wp = ((W + X - 1) / X) * X;
    return 2 * (size_t)((Mp + Wp + Mp) / X * (X + 1)) * G * sizeof(float2) +
           2 * (size_t)demig_idx_words(Wp, Mp) * sizeof(unsigned);
}

static const ClusterKernel *find_cluster(int L)
{
    for (const auto &k : kCluster)
        if (k.L == L) return &k;
    return nullptr;
}

// ---------------------------------------------------------------------------------------
// Naive comparison kernel: one launch per (shot, frequency, depth), one thread per position,
// wavefields and operators in global memory.
// ---------------------------------------------------------------------------------------
__global__ void naive_step_kernel(const float4 *__restrict__ cur, float4 *__restrict__ nxt, int w,
                                  int M, const cpx *__restrict__ tab, int tab_stride,
                                  const uint16_t *__restrict__ idx_row, int x0,
                                  float *__restrict__ image_row)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w) return;
    const cpx *t = tab + (long long)idx_row[x0 + i] * tab_stride;
    float sr = 0.f, si = 0.f, rr = 0.f, ri = 0.f;
    for (int k = 0; k <= 2 * M; ++k) {
        const float4 v = cur[i + k];
        const cpx f = t[k];
        sr = fmaf(f.re, v.x, sr); sr = fmaf(-f.im, v.y, sr);
        si = fmaf(f.re, v.y, si); si = fmaf(f.im, v.x, si);
        rr = fmaf(f.re, v.z, rr); rr = fmaf(-f.im, v.w, rr);
        ri = fmaf(f.re, v.w, ri); ri = fmaf(f.im, v.z, ri);
    }
    nxt[i + M] = make_float4(sr, si, rr, ri);
    atomicAdd(image_row + x0 + i, sr * rr - si * ri);
}

__global__ void naive_pack_kernel(const cpx *__restrict__ wave, const cpx *__restrict__ shot, int w,
                                  int M, float4 *__restrict__ buf, int to_buf)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w) return;
    if (to_buf) {
        const cpx S = wave[i], R = shot[i];
        buf[i + M] = make_float4(S.re, S.im, R.re, -R.im);
    }
}

__global__ void naive_unpack_kernel(const float4 *__restrict__ buf, int w, int M,
                                    cpx *__restrict__ wave, cpx *__restrict__ shot)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w) return;
    const float4 v = buf[i + M];
    wave[i] = cpx{v.x, v.y};
    shot[i] = cpx{v.z, -v.w};
}

// Dense operator table of the reference's legacy ABI from the compact table and the operator index:
// dense[l][j][x][k] = tab[idx[j][l][x]][k] (conjugated when conj != 0).  One block per (l, j) row of
// nx*L elements, written with coalesced stores; x and k advance incrementally with the block stride.
__global__ void dense_table_kernel(const uint16_t *__restrict__ idx, int nf, int nextrap, int nx, int lstride,
                                   const cpx *__restrict__ tab, int tab_stride, int L, int conj,
                                   cpx *__restrict__ dense)
{
    const int lj = blockIdx.x;  // l * nf + j
    const int l = lj / nf, j = lj - l * nf;
    const uint16_t *irow = idx + ((long long)j * nextrap + l) * lstride;
    cpx *out = dense + (long long)lj * nx * L;
    const int n = nx * L;
    const int sx = (int)blockDim.x / L, sk = (int)blockDim.x - sx * L;
    int x = (int)threadIdx.x / L, k = (int)threadIdx.x - x * L;
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
        cpx v = tab[(long long)irow[x] * tab_stride + k];
        if (conj) v.im = -v.im;
        out[e] = v;
        x += sx;
        k += sk;
        if (k >= L) {
            k -= L;
            ++x;
        }
    }
}

// L2 read probe: every thread streams float4 from an L2-resident buffer with ld.global.cg (L2 only,
// no L1 allocation); four independent accumulators keep many loads in flight.
__global__ void l2_read_probe_kernel(const float4 *__restrict__ buf, long long n4, int iters, float *out)
{
    float4 acc[4] = {};
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    for (int it = 0; it < iters; ++it) {
        long long i = t0;
        for (; i + 3 * stride < n4; i += 4 * stride) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float4 v = __ldcg(buf + i + u * stride);
                acc[u].x += v.x; acc[u].y += v.y; acc[u].z += v.z; acc[u].w += v.w;
            }
        }
        for (; i < n4; i += stride) {
            const float4 v = __ldcg(buf + i);
            acc[0].x += v.x; acc[0].y += v.y; acc[0].z += v.z; acc[0].w += v.w;
        }
    }
    float s = 0.f;
#pragma unroll
    for (int u = 0; u < 4; ++u) s += acc[u].x + acc[u].y + acc[u].z + acc[u].w;
    out[t0] = s;
}

// FP32 FMA probe: 16 independent chains per thread so the FMA pipe, not latency, limits it.
__global__ void fma_probe_kernel(float *out, int iters)
{
    float a[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) a[i] = threadIdx.x * 1e-3f + i;
    const float b = 0.9999f, c = 1e-4f;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
            for (int i = 0; i < 16; ++i) a[i] = fmaf(a[i], b, c);
    }
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) s += a[i];
    out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

// ---------------------------------------------------------------------------------------
// Device allocation.  Every device buffer the library allocates goes through device_alloc, which
// refuses (IMG2D_ENOMEM, before calling cudaMalloc) any single allocation larger than the limit set
// by img2d_set_alloc_limit or, until that is called, by the environment variable
// IMG2D_ALLOC_LIMIT_BYTES (unset or 0: no limit).  The limit injects allocation failures on the
// host for tests of the error path, including through the void drop-in shims.
// ---------------------------------------------------------------------------------------
static std::mutex g_alloc_mu;
static bool g_alloc_limit_set = false;
static size_t g_alloc_limit = 0;

static size_t alloc_limit()
{
    std::lock_guard<std::mutex> lock(g_alloc_mu);
    if (!g_alloc_limit_set) {
        const char *e = getenv("IMG2D_ALLOC_LIMIT_BYTES");
        g_alloc_limit = e ? (size_t)strtoull(e, nullptr, 10) : 0;
        g_alloc_limit_set = true;
    }
    return g_alloc_limit;
}

// Device blocks given back by plans and host calls, kept for the next allocation of about their size (up
// to 2 GB a device; img2d_release_host_cache frees them, and so does an allocation that finds no
// memory).  cudaMalloc and cudaFree of the large buffers cost milliseconds: the planes of a
// demigration of 5 shots (0.6 GB) 13 ms, the tables of a dense call (0.25 GB) 3 ms.  A block enters
// only after the device has finished its work (cudaFree waits for the same), so whoever takes it, on
// any stream or thread, finds nobody using it.
constexpr size_t kPoolMaxBytes = 2ull << 30, kPoolMinBlock = 256 << 10;
struct DevicePool {
    std::mutex mu;
    std::map<int, std::multimap<size_t, void *>> blocks;  // per device, by size
    std::map<int, size_t> bytes;
};
static DevicePool &device_pool()
{
    static DevicePool *pool = new DevicePool;  // never destroyed: static objects give buffers back at exit
    return *pool;
}

static void pool_flush(int dev)
{
    DevicePool &pool = device_pool();
    std::lock_guard<std::mutex> lock(pool.mu);
    for (auto &b : pool.blocks[dev]) cudaFree(b.second);
    pool.blocks[dev].clear();
    pool.bytes[dev] = 0;
}

// n bytes on the current device; *got: the size of the block, for device_free.
static int device_alloc(void **p, size_t n, size_t *got, int *dev)
{
    *p = nullptr;
    *got = n;
    *dev = 0;
    const size_t lim = alloc_limit();
    if (lim && n > lim)
        return fail(IMG2D_ENOMEM, "device allocation of " + std::to_string(n) + " bytes refused: above the " +
                                      std::to_string(lim) + "-byte allocation limit (IMG2D_ALLOC_LIMIT_BYTES)");
    if (cudaGetDevice(dev) != cudaSuccess) cudaGetLastError();
    if (n >= kPoolMinBlock) {
        DevicePool &pool = device_pool();
        std::lock_guard<std::mutex> lock(pool.mu);
        auto &blocks = pool.blocks[*dev];
        auto it = blocks.lower_bound(n);
        if (it != blocks.end() && it->first <= n + n / 4) {
            *p = it->second;
            *got = it->first;
            pool.bytes[*dev] -= it->first;
            blocks.erase(it);
            return IMG2D_OK;
        }
    }
    cudaError_t e = cudaMalloc(p, n);
    if (e != cudaSuccess) {
        cudaGetLastError();
        pool_flush(*dev);
        e = cudaMalloc(p, n);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
        return fail(IMG2D_ENOMEM, "cudaMalloc(" + std::to_string(n) + " bytes): " + cudaGetErrorString(e));
    }
    return IMG2D_OK;
}

// Waits for the work of all streams of the current device, as cudaFree of the block itself would: a
// cudaFree of a small one.  cudaDeviceSynchronize would invalidate a capture that is going on in a
// stream of the device (in another thread, or in this one in relaxed mode), where freeing is allowed.
static bool wait_as_free_does()
{
    void *q = nullptr;
    return cudaMalloc(&q, 256) == cudaSuccess && cudaFree(q) == cudaSuccess;
}

static void device_free(void *p, size_t n, int dev)
{
    int cur = -1;
    if (n >= kPoolMinBlock && n <= kPoolMaxBytes && cudaGetDevice(&cur) == cudaSuccess && cur == dev && wait_as_free_does()) {
        DevicePool &pool = device_pool();
        std::lock_guard<std::mutex> lock(pool.mu);
        try {
            if (pool.bytes[dev] + n <= kPoolMaxBytes) {
                pool.blocks[dev].emplace(n, p);
                pool.bytes[dev] += n;
                return;
            }
        } catch (...) {  // no host memory for the entry: the block is freed
        }
    }
    cudaGetLastError();
    cudaFree(p);
}

// Pinned staging for uploads from pageable memory.  A plain cudaMemcpy of pageable memory runs at the
// speed of one host thread (about 10 GB/s here); four workers copying 2 MB pieces into a pinned ring,
// each sending its own, reach 34 GB/s (eight 31, sixteen 22).  One upload uses the ring at a time,
// others take the plain copy.  The ring (16 MB) is kept until img2d_release_host_cache.
constexpr size_t kStagePiece = 2 << 20;
constexpr int kStageWorkers = 4;
struct StageRing {
    std::mutex mu;
    unsigned char *host = nullptr;
};
static StageRing &stage_ring()
{
    static StageRing *r = new StageRing;
    return *r;
}

// One piece of an upload; the pieces of group g are issued before those of group g + 1.
struct UploadPiece {
    void *dst;
    const void *src;
    size_t n;
    int group;
};

static void add_pieces(std::vector<UploadPiece> &v, void *dst, const void *src, size_t n, int group)
{
    for (size_t at = 0; at < n; at += kStagePiece)
        v.push_back({(unsigned char *)dst + at, (const unsigned char *)src + at, std::min(kStagePiece, n - at), group});
}

// Host to device on stream st.  ready(g) runs on the calling thread once every piece of group g is queued
// on st; returns when all copies have completed.  The workers live for the whole call: a new thread's
// first CUDA call costs a tenth of a millisecond, as much as two pieces.
static int upload(const std::vector<UploadPiece> &pieces, int groups, cudaStream_t st, const std::function<int(int)> &ready)
{
    size_t total = 0;
    for (const UploadPiece &u : pieces) total += u.n;
    // staged from pageable memory only, every array of the first group: the workers copy on the host
    bool staged = total >= 4 * kStagePiece;
    const unsigned char *next_src = nullptr;
    for (size_t i = 0; staged && i < pieces.size() && pieces[i].group == pieces[0].group; ++i) {
        cudaPointerAttributes at{};
        if (pieces[i].src != next_src && cudaPointerGetAttributes(&at, pieces[i].src) == cudaSuccess)
            staged = at.type == cudaMemoryTypeUnregistered;
        next_src = (const unsigned char *)pieces[i].src + pieces[i].n;
    }
    cudaGetLastError();
    StageRing &ring = stage_ring();
    std::unique_lock<std::mutex> lock(ring.mu, std::defer_lock);
    staged = staged && lock.try_lock();
    if (staged && !ring.host &&
        cudaHostAlloc((void **)&ring.host, 2 * kStageWorkers * kStagePiece, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        ring.host = nullptr;
        staged = false;
    }
    int dev = 0, rc = IMG2D_OK;
    IMG2D_CUDA(cudaGetDevice(&dev));
    std::mutex mu;
    std::condition_variable cv;
    std::vector<size_t> left(groups, 0);  // pieces of a group not yet queued
    for (const UploadPiece &u : pieces) ++left[u.group];
    size_t next = 0;
    cudaError_t err = cudaSuccess;
    auto work = [&](int w) {
        cudaError_t e = cudaSetDevice(dev);
        cudaEvent_t ev[2] = {nullptr, nullptr};
        for (int i = 0; i < 2 && e == cudaSuccess; ++i) e = cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming);
        std::unique_lock<std::mutex> l(mu);
        for (int k = 0; e == cudaSuccess && err == cudaSuccess && next < pieces.size(); ++k) {
            const UploadPiece u = pieces[next++];
            l.unlock();
            unsigned char *slot = ring.host + (size_t)(2 * w + (k & 1)) * kStagePiece;
            if (k >= 2) e = cudaEventSynchronize(ev[k & 1]);  // the slot's previous piece has left
            if (e == cudaSuccess) {
                std::memcpy(slot, u.src, u.n);
                e = cudaMemcpyAsync(u.dst, slot, u.n, cudaMemcpyHostToDevice, st);
            }
            if (e == cudaSuccess) e = cudaEventRecord(ev[k & 1], st);
            l.lock();
            if (e == cudaSuccess && --left[u.group] == 0) cv.notify_one();
        }
        if (e != cudaSuccess) err = e;
        cv.notify_one();
        l.unlock();
        for (cudaEvent_t x : ev)
            if (x) cudaEventDestroy(x);
    };
    std::vector<std::thread> threads;
    if (staged) {
        try {
            threads.reserve(kStageWorkers);
            for (int w = 0; w < kStageWorkers; ++w) threads.emplace_back(work, w);
        } catch (...) {
            if (threads.empty()) staged = false;  // fewer workers do as well
        }
    }
    size_t plain = 0;
    for (int g = 0; g < groups && !rc; ++g) {
        if (staged) {
            std::unique_lock<std::mutex> l(mu);
            cv.wait(l, [&]() { return left[g] == 0 || err != cudaSuccess; });
            if (err != cudaSuccess) break;
        } else {
            for (; plain < pieces.size() && pieces[plain].group == g && err == cudaSuccess; ++plain)
                err = cudaMemcpyAsync(pieces[plain].dst, pieces[plain].src, pieces[plain].n, cudaMemcpyHostToDevice, st);
            if (err != cudaSuccess) break;
        }
        rc = ready(g);
    }
    if (rc) {
        std::lock_guard<std::mutex> l(mu);
        next = pieces.size();
    }
    for (std::thread &t : threads) t.join();
    const cudaError_t done = cudaStreamSynchronize(st);  // also before the ring has its next user
    if (rc) return rc;
    IMG2D_CUDA(err);
    IMG2D_CUDA(done);
    return IMG2D_OK;
}

// ---------------------------------------------------------------------------------------
// Plan
// ---------------------------------------------------------------------------------------
// Bump allocator over a fixed device region (the no-allocation entry point's static scratch).
struct Carver {
    unsigned char *base = nullptr;
    size_t cap = 0, used = 0;
};

struct DevBuf {
    void *p = nullptr;
    size_t bytes = 0;
    bool owned = false;
    int dev = 0;               // device of an owned block
    Carver *carver = nullptr;  // when set, storage is carved from it and never freed
    ~DevBuf() { release(); }
    void release()
    {
        if (p && owned) device_free(p, bytes, dev);
        p = nullptr;
        bytes = 0;
        owned = false;
    }
    int ensure(size_t n)
    {
        if (n <= bytes && p) return IMG2D_OK;
        release();
        if (carver) {
            const size_t off = (carver->used + 255) & ~(size_t)255;
            if (off + n > carver->cap)
                return fail(IMG2D_EINVAL, "problem needs more than the " + std::to_string(carver->cap >> 20) +
                                              " MiB of fixed scratch of the no-allocation entry point");
            p = carver->base + off;
            bytes = n;
            carver->used = off + n;
            return IMG2D_OK;
        }
        if (n == 0) n = 16;
        size_t got = 0;
        const int rc = device_alloc(&p, n, &got, &dev);
        if (rc) return rc;
        owned = true;
        bytes = got;
        return IMG2D_OK;
    }
    template <class T> T *as() const { return static_cast<T *>(p); }
};

}  // namespace img2d

struct img2d_plan {
    int ns = 0, nextrap = 0, nz = 0, nx = 0, nf = 0, nt = 0, M = 0, L = 0, nk = 0, flags = 0;
    int mode = img2d::OP_CONJ;
    int G = 1, grid = 0, n_items = 0, max_w = 0, tab_stride = 0, idx_lstride = 0;
    bool fixed = false;
    img2d::KernelFn fn = nullptr;
    size_t smem = 0;
    std::vector<int> x0, w;
    std::vector<long long> off;
    long long wave_elems = 0;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    bool ev_recorded = false;
    bool launched = false;  // a kernel that reports to the status word, or could, has been queued
    // identity of this plan for caches keyed on it (a new plan may reuse a freed plan's address)
    const unsigned long long uid = next_uid();
    static unsigned long long next_uid()
    {
        static std::atomic<unsigned long long> n{0};
        return ++n;
    }
    const char *packing = "lines";  // how shots were packed into the wide kernel's items
    double pack_cost = 0.0;         // wide kernel: modelled cost of all items of one frequency, in CTA units
    double computed_per_useful = 0.0;  // computed (slot, position) pairs per aperture sample
    ~img2d_plan()
    {
        if (ev0) cudaEventDestroy(ev0);
        if (ev1) cudaEventDestroy(ev1);
    }
    int n_slots = 0;
    std::vector<int> group_order;  // migration groups, widest first (the order of the item queue)
    int cluster = 0;  // CTAs per cluster of the cluster kernel, 0 = single-CTA kernels
    int block = 256;                  // threads per CTA of the chosen kernel
    bool rows_tab_set = false;        // tab_rows holds the tables of the last set_model
    bool rows = false;                // the row-split kernel (its table order, visit counts per CTA)
    img2d::RowsStarts row_starts{{0, 0, 0, 0}, 0, 0.0};  // set by plan_row_starts on its first call
    int variant = -1;                 // index into the cluster2 variant table
    int tab16 = 0;                    // operator table storage: 0 FP32, 1 FP16, 2 BF16
    const char *kname = "";           // name of the chosen kernel
    img2d::Carver *carver = nullptr;  // no-allocation mode: buffers carved from fixed scratch
    cudaStream_t upload_stream = 0;   // no-allocation mode: stream of the descriptor uploads
    bool timing = true;               // record events around the migration kernel
    img2d::DevBuf items, groups, segs, owner, shot_off, idx, tabF, tabB, tab16buf, tab_rows, partial, comp, visits, counter, naive_buf;
    // dense tables (drop-in ABI) are owned by the caller of run_dense
    // lane-slot packing: shots of each slot, slots ordered by extent, right end of each slot
    std::vector<std::vector<int>> slots;
    std::vector<int> slot_order, slot_end;
    // demigration (adjoint) launch state, built on its first call
    int adj_G = 0, adj_grid = 0, adj_items_n = 0, adj_wmax = 0, adj_block = 0, adj_slab = 0, adj_nslab = 0;
    int adj_cluster = 0;               // CTAs per cluster of the cluster demigration kernel, 0 = single CTA
    bool adj_rows = false;             // the row-split demigration kernel
    bool adj_allow_rows = true, adj_allow_wide = true;  // until their planes did not fit in memory
    void (*adj_rows_fn)(img2d::RowsAdjArgs) = nullptr;
    void (*adj_wide_fn)(img2d::DemigrateArgs, int *) = nullptr;  // the wide demigration kernel
    bool adj_full_cache = false;       // kept source: every depth step of every item (else per-CTA planes only)
    bool adj_ring = false;             // its forward steps read operator pairs through the shared-memory ring
    bool model_set = false;            // set_model has built the padded tables and the operator index
    long long adj_work_cta = 0, adj_cache_item = 0;  // float2 elements: per-CTA work area, kept per item
    size_t adj_smem = 0;
    void (*adj_fn)(img2d::DemigrateArgs) = nullptr;
    img2d::DevBuf adj_items, adj_groups, adj_segs, adj_owner, adj_work, adj_counter;
    img2d::DevBuf adj_cache;   // source checkpoints kept per item (IMG2D_SOURCE_KEEP)
    bool adj_cache_valid = false;
};

namespace img2d {

static int check_device()
{
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n == 0) {
        cudaGetLastError();
        return fail(IMG2D_ENODEV, "no CUDA device visible to imaging2d_wlsq_b200");
    }
    return IMG2D_OK;
}

// Largest portable cluster is 8 CTAs; B200 runs up to 16 when the kernel opts in.
constexpr int kMaxCluster = 16;

// How many clusters of K CTAs (block threads, smem bytes each) of `fn` fit on the device at once;
// 0 when none does.  K > 8 sets the non-portable cluster-size attribute first.
static int clusters_that_fit(const void *fn, int K, int block, size_t smem)
{
    if (K > 8 && cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = K;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.gridDim = dim3(K * 64, 1, 1);
    cfg.blockDim = dim3(block, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

// Shared memory bytes of one CTA for groups of G shots over a union window of width W.
static size_t smem_bytes(int G, int W, int M, int X)
{
    const int Mp = ((M + X - 1) / X) * X;
    const int Wp = ((W + X - 1) / X) * X;
    const int npos = Mp + Wp + Mp;
    const size_t nslot = (size_t)npos / X * (X + 1);
    return 2 * nslot * G * sizeof(float4);
}

// One group from its lines (each a list of shots, in increasing x, separated by >= M zero samples).
static void emit_group(const img2d_plan *p, const std::vector<std::vector<int>> &lines, std::vector<GroupDesc> &groups,
                       std::vector<int4> &segs, std::vector<int16_t> &owner)
{
    int u0 = p->nx, u1 = 0;
    for (const auto &line : lines)
        for (int s : line) {
            u0 = std::min(u0, p->x0[s]);
            u1 = std::max(u1, p->x0[s] + p->w[s]);
        }
    GroupDesc gd{};
    gd.seg_begin = (int)segs.size();
    gd.u0 = u0;
    gd.W = u1 - u0;
    gd.nslots = (int)lines.size();
    gd.owner_stride = (gd.W + 7) / 8 * 8;
    gd.owner_off = (long long)owner.size();
    owner.resize(owner.size() + (size_t)gd.nslots * gd.owner_stride, (int16_t)-1);
    for (int k = 0; k < gd.nslots; ++k)
        for (int s : lines[k]) {
            segs.push_back(make_int4(s, k, p->x0[s], p->w[s]));
            int16_t *row = owner.data() + gd.owner_off + (size_t)k * gd.owner_stride;
            for (int x = p->x0[s]; x < p->x0[s] + p->w[s]; ++x) row[x - u0] = (int16_t)s;
        }
    gd.nseg = (int)segs.size() - gd.seg_begin;
    groups.push_back(gd);
}

// Slots of similar extent form groups of G that share a work item; returns the widest group.
static int pack_groups(const img2d_plan *p, int G, std::vector<GroupDesc> &groups, std::vector<int4> &segs,
                       std::vector<int16_t> &owner)
{
    groups.clear();
    segs.clear();
    owner.clear();
    int widest = 0;
    const std::vector<int> &sorder = p->slot_order;
    for (size_t g0 = 0; g0 < sorder.size(); g0 += G) {
        const int n = (int)std::min<size_t>(G, sorder.size() - g0);
        std::vector<std::vector<int>> lines;
        for (int k = 0; k < n; ++k) lines.push_back(p->slots[sorder[g0 + k]]);
        emit_group(p, lines, groups, segs, owner);
        widest = std::max(widest, groups.back().W);
    }
    return widest;
}

// Wide kernel (8 slots x 1024 positions per CTA, clusters of K CTAs, each item's window split
// evenly over the cluster in 256-position units): cost of one item of width W in CTA units (one
// CTA, one depth step, all 1024 positions), divided by the throughput of a CTA with NC/64 busy
// warps relative to 16.  The relative throughputs were measured on a B200 on equal work (full
// aperture shots, windows of 2048/1536/512/256 positions): 0.92 with 12 busy warps, 0.87 with 8,
// 0.62 with 4.  eff12 replaces the 12-warp figure (the packing's greedy also tries other values to
// steer its choices; costs are always compared with the measured one).
static double wide_item_cost(int W, int K, double eff12 = 0.92)
{
    const int NC = std::min(WideShape::PC, (W + K * 256 - 1) / (K * 256) * 256);
    const double eff = NC >= 1024 ? 1.0 : (NC >= 768 ? eff12 : (NC >= 512 ? 0.87 : 0.62));
    return (double)K * NC / WideShape::PC / eff;
}

// The shots of `pool` (sorted by aperture end) that lie inside [u0, u1), in that order; returns
// their total aperture width.
static long long window_shots(const img2d_plan *p, const std::vector<int> &pool, int u0, int u1,
                              std::vector<int> &cand)
{
    cand.clear();
    long long sum = 0;
    for (int s : pool)
        if (p->x0[s] >= u0 && p->x0[s] + p->w[s] <= u1) {
            cand.push_back(s);
            sum += p->w[s];
        }
    return sum;
}

// Up to G lines from the shots `cand` (sorted by aperture end): each line is the heaviest chain of
// shots (total aperture width) separated by >= M, taken in turn (weighted interval scheduling,
// repeated).  Returns the aperture width covered; the lines when asked.
static long long window_lines(const img2d_plan *p, std::vector<int> cand, int G,
                              std::vector<std::vector<int>> *lines_out)
{
    long long covered = 0;
    std::vector<long long> best, ends;
    std::vector<int> prev;
    std::vector<char> take;
    for (int line = 0; line < G && !cand.empty(); ++line) {
        const int n = (int)cand.size();
        ends.resize(n);
        best.assign(n + 1, 0);
        prev.resize(n);
        take.assign(n, 0);
        for (int i = 0; i < n; ++i) ends[i] = (long long)p->x0[cand[i]] + p->w[cand[i]] + p->M;
        for (int i = 0; i < n; ++i) {
            const int s = cand[i];
            // shots before i that end (with the M gap) at or before this one's start
            const int j = (int)(std::upper_bound(ends.begin(), ends.begin() + i, (long long)p->x0[s]) - ends.begin());
            prev[i] = j;
            const long long with = best[j] + p->w[s];
            if (with > best[i]) {
                best[i + 1] = with;
                take[i] = 1;
            } else {
                best[i + 1] = best[i];
            }
        }
        std::vector<int> chosen;
        std::vector<char> used(n, 0);
        for (int i = n; i > 0;) {
            if (take[i - 1]) {
                chosen.push_back(cand[i - 1]);
                used[i - 1] = 1;
                i = prev[i - 1];
            } else {
                --i;
            }
        }
        covered += best[n];
        if (lines_out) {
            std::reverse(chosen.begin(), chosen.end());
            lines_out->push_back(chosen);
        }
        std::vector<int> rest;
        for (int i = 0; i < n; ++i)
            if (!used[i]) rest.push_back(cand[i]);
        cand.swap(rest);
    }
    return covered;
}

// Window-first packing for the wide kernel: repeatedly take the window (a start on a 32-position
// grid or at an end of one of the 8 widest remaining shots, and a width of K x 256 x m positions,
// m = 1..4, the widths at which an item's cost steps) whose G best lines of the remaining shots
// cover the most aperture per unit of cost, until every shot is placed.  Narrow windows become narrow items, which the kernel runs with fewer busy warps
// instead of computing positions outside every aperture.  Returns the total cost in CTA units.
static double pack_groups_windows(const img2d_plan *p, int G, int K, std::vector<GroupDesc> &groups,
                                  std::vector<int4> &segs, std::vector<int16_t> &owner, double sel_eff12 = 0.92)
{
    groups.clear();
    segs.clear();
    owner.clear();
    std::vector<int> pool(p->ns);
    std::iota(pool.begin(), pool.end(), 0);
    std::stable_sort(pool.begin(), pool.end(),
                     [&](int a, int b) { return p->x0[a] + p->w[a] < p->x0[b] + p->w[b]; });
    const int nx = p->nx;
    const int step = std::max(32, (nx / 64 + 31) / 32 * 32);
    double total = 0.0;
    std::vector<int> starts, cand, prev;
    while (!pool.empty()) {
        double best_ratio = -1.0;
        int best_u0 = 0, best_w = 0;
        // the 8 widest remaining shots also get windows aligned to either of their ends, so that a
        // shot nearly as wide as a window still has one that holds it
        std::vector<int> widest(pool);
        std::stable_sort(widest.begin(), widest.end(), [&](int a, int b) { return p->w[a] > p->w[b]; });
        widest.resize(std::min<size_t>(8, widest.size()));
        for (int m = 1; m <= 4; ++m) {
            const int W = std::min(nx, K * 256 * m);
            const double c = wide_item_cost(W, K, sel_eff12);
            starts.clear();
            for (int u = 0; u <= std::max(nx - W, 0) + step - 1; u += step) starts.push_back(u);
            for (int s : widest) starts.push_back(p->x0[s]);
            for (int s : widest) starts.push_back(p->x0[s] + p->w[s] - W);
            prev.clear();
            for (int u : starts) {
                const int u0 = std::max(0, std::min(u, nx - W));
                // the total width of the shots inside bounds what G lines can cover; a window with
                // the same shots as the previous one of this width covers the same
                const long long bound = window_shots(p, pool, u0, u0 + W, cand);
                if (bound == 0 || bound / c <= best_ratio || cand == prev) continue;
                prev = cand;
                const long long cov = window_lines(p, cand, G, nullptr);
                if (cov > 0 && cov / c > best_ratio) {
                    best_ratio = cov / c;
                    best_u0 = u0;
                    best_w = W;
                }
            }
            if (W >= nx) break;
        }
        if (best_ratio <= 0.0) return -1.0;  // a shot wider than every window (not reached: K covers it)
        std::vector<std::vector<int>> lines;
        window_shots(p, pool, best_u0, best_u0 + best_w, cand);
        window_lines(p, cand, G, &lines);
        emit_group(p, lines, groups, segs, owner);
        total += wide_item_cost(groups.back().W, K);
        std::vector<char> placed(p->ns, 0);
        for (const auto &line : lines)
            for (int s : line) placed[s] = 1;
        std::vector<int> rest;
        for (int s : pool)
            if (!placed[s]) rest.push_back(s);
        pool.swap(rest);
    }
    return total;
}

// Pack shots into lane slots: shots sorted by aperture start go to the slot whose last shot ends
// furthest to the left while still leaving >= M zero samples before this one (interval colouring,
// best fit); full-aperture shots get a slot each.  Slots are then ordered by extent.  Needs x0, w
// and M of the plan.
static void colour_slots(img2d_plan *p)
{
    const int ns = (int)p->x0.size(), M = p->M;
    std::vector<int> order(ns);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        if (p->x0[a] != p->x0[b]) return p->x0[a] < p->x0[b];
        return p->w[a] < p->w[b];
    });
    std::vector<std::vector<int>> slots;
    std::vector<int> slot_end;
    for (int s : order) {
        int best = -1;
        for (size_t i = 0; i < slots.size(); ++i)
            if (slot_end[i] + M <= p->x0[s] && (best < 0 || slot_end[i] > slot_end[best])) best = (int)i;
        if (best < 0) {
            slots.push_back({s});
            slot_end.push_back(p->x0[s] + p->w[s]);
        } else {
            slots[best].push_back(s);
            slot_end[best] = p->x0[s] + p->w[s];
        }
    }
    std::vector<int> sorder(slots.size());
    std::iota(sorder.begin(), sorder.end(), 0);
    auto ext0 = [&](int i) { return p->x0[slots[i].front()]; };
    std::stable_sort(sorder.begin(), sorder.end(), [&](int a, int b) {
        if (ext0(a) != ext0(b)) return ext0(a) < ext0(b);
        return slot_end[a] < slot_end[b];
    });
    p->n_slots = (int)slots.size();
    p->slots = slots;
    p->slot_order = sorder;
    p->slot_end = slot_end;
}

// Surveys with more shots keep the line packing: the window greedy would take seconds per plan.
constexpr int kWindowPackingMaxShots = 2048;

// The window-first packing with three weightings of 12-warp items in the greedy's choices (the
// measured 0.92, then 0.95 and 1.0: a myopic greedy lands on different packings); keeps the one of
// lowest measured-model cost.  The greedy's time grows about as the square of the shot count
// (0.4 s for 1024 shots on one host core), so above 512 shots only the measured weighting runs.
static double pack_windows_best(const img2d_plan *p, int G, int K, std::vector<GroupDesc> &groups,
                                std::vector<int4> &segs, std::vector<int16_t> &owner)
{
    double best = -1.0;
    const double sels[3] = {0.92, 0.95, 1.0};
    const int nsel = p->ns > 512 ? 1 : 3;
    for (int i = 0; i < nsel; ++i) {
        const double sel = sels[i];
        std::vector<GroupDesc> g2;
        std::vector<int4> s2;
        std::vector<int16_t> o2;
        const double c = pack_groups_windows(p, G, K, g2, s2, o2, sel);
        if (c > 0.0 && (best < 0.0 || c < best - 1e-9)) {
            best = c;
            groups.swap(g2);
            segs.swap(s2);
            owner.swap(o2);
        }
    }
    return best;
}

// The search takes 10 to 550 us on the host: once per plan, not at every launch.
static const RowsStarts &plan_row_starts(img2d_plan *p)
{
    if (!p->row_starts.apart) p->row_starts = rows_starts(p->L);
    return p->row_starts;
}

static int build_plan(img2d_plan *p, int ns, int nextrap, int nz, int nx, int nf, int nt, int M,
                      int nk, const int *shot_x0, const int *shot_nx, int flags, int mode)
{
    if (ns <= 0 || nextrap <= 0 || nz < nextrap || nx <= 0 || nf <= 0 || nt < nf || M < 0)
        return fail(IMG2D_EINVAL, "invalid dimensions (need ns>0, 0<nextrap<=nz, nx>0, 0<nf<=nt, M>=0)");
    if (mode != OP_DENSE && (nk <= 0 || nk > 65535))
        return fail(IMG2D_EINVAL, "nk must be in [1, 65535]");
    if ((long long)nf * nextrap * nx > (1ll << 40)) return fail(IMG2D_EINVAL, "problem too large");
    if (ns > 32767) return fail(IMG2D_EINVAL, "at most 32767 shots per plan");
    p->ns = ns; p->nextrap = nextrap; p->nz = nz; p->nx = nx; p->nf = nf; p->nt = nt; p->M = M;
    p->L = 2 * M + 1; p->nk = nk; p->flags = flags; p->mode = mode;
    p->x0.assign(ns, 0);
    p->w.assign(ns, nx);
    for (int s = 0; s < ns; ++s) {
        if (shot_x0) p->x0[s] = shot_x0[s];
        if (shot_nx) p->w[s] = shot_nx[s];
        if (p->x0[s] < 0 || p->w[s] <= 0 || p->x0[s] + p->w[s] > nx)
            return fail(IMG2D_EINVAL, "shot " + std::to_string(s) + " aperture outside [0, nx)");
    }
    p->off.assign(ns, 0);
    long long acc = 0;
    for (int s = 0; s < ns; ++s) {
        p->off[s] = acc;
        acc += (long long)nt * p->w[s];
    }
    p->wave_elems = acc;

    int dev = 0;
    IMG2D_CUDA(cudaGetDevice(&dev));
    int smem_optin = 0, nsm = 0;
    IMG2D_CUDA(cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    IMG2D_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const int static_reserve = 1024;

    colour_slots(p);

    std::vector<GroupDesc> groups;
    std::vector<int4> segs;
    std::vector<int16_t> owner;
    auto make_groups = [&](int G) { return pack_groups(p, G, groups, segs, owner); };

    // Kernel choice, for 7 taps and more.  8 slots: the wide kernel (try_wide) where the 16-slot kernels'
    // clusters would leave SMs idle or there are 6 to 11 slots.  16 slots: the same kernel with 8 lanes
    // per group (try_wide16, up to 65 taps), else the second-generation cluster kernel, else the
    // first-generation one (256 positions per CTA, up to 8 CTAs, compile-time lengths).  The row-split
    // kernel for table pairs, fewer than 6 slots, and where it is estimated faster than any of these.
    // Otherwise the single-CTA kernels with the largest power of two <= 8 slots whose ping-pong
    // buffers fit in shared memory.
    p->cluster = 0;
    p->block = 256;
    const bool cluster_ok = mode == OP_CONJ && !(flags & (IMG2D_FLAG_GENERIC | IMG2D_FLAG_NO_CLUSTER)) &&
                            p->n_slots >= 12;
    int vsel = (flags >> IMG2D_FLAG_VARIANT_SHIFT) & 0xff;
    const bool explicit_variant = vsel >= 1 && vsel <= kNumCluster2;
    vsel = explicit_variant ? vsel - 1 : kCluster2Default;
    Cluster2Variant cv = kCluster2[vsel];
    const int tab16 = (flags & IMG2D_FLAG_TABLE_BF16) ? 2 : ((flags & IMG2D_FLAG_TABLE_FP16) ? 1 : 0);
    if (tab16) {
        // reduced-precision operator storage: the staged shape with 16-bit tap loads
        cv = {16, false, false,
              tab16 == 1 ? migrate_cluster2_kernel<16, false, false, false, TAB_F16, 4>
                         : migrate_cluster2_kernel<16, false, false, false, TAB_BF16, 4>,
              true};
        vsel = kCluster2Staged;
    }
    // Use variant v when its shared memory fits and, for windows wider than 8 CTAs, clusters of the
    // needed size fit on the device.
    auto try_cluster2 = [&](const Cluster2Variant &v, int index) {
        const int pc2 = v.nw * 32;
        const size_t smem2 = cluster2_smem_bytes(M, pc2) + (v.stage ? cluster2_stage_bytes(pc2) : 0) +
                             (v.ring ? cluster2_ring_bytes(pc2) : 0);
        if (smem2 + static_reserve > (size_t)smem_optin) return false;
        const int widest = make_groups(16);
        const int K = (widest + pc2 - 1) / pc2;
        if (!(K <= 8 || (K <= kMaxCluster && clusters_that_fit((const void *)v.fn, K, pc2, smem2) > 0))) return false;
        p->cluster = K;
        p->G = 16;
        p->fixed = true;
        p->fn = v.fn;
        p->smem = smem2;
        p->max_w = widest;
        p->block = pc2;
        p->variant = index;
        p->kname = "migrate_cluster2";
        return true;
    };
    // Wide cluster kernel (8 slots x 1024 positions per CTA, clusters of half the size, packed FMAs).
    // It is the default where the cluster2 kernel's clusters would leave SMs idle (clusters of 4 fit
    // 33 times on 148 SMs), and on request (IMG2D_FLAG_WIDE / _WIDE_SCALAR).
    auto try_wide = [&]() {
        // with the step-ahead stage where its 12 KB fit (operators up to 49 taps); the bulk-copy
        // ring adds 256 bytes of barriers
        const bool bulk = (flags & IMG2D_FLAG_WIDE_BULK) != 0;
        const size_t bars = bulk ? wide_bulk_smem_bytes(M, true) - wide_stage_smem_bytes(M) : 0;
        const bool stage = wide_stage_smem_bytes(M) + bars + static_reserve <= (size_t)smem_optin;
        KernelFn wf;
        if (bulk)
            wf = stage ? migrate_wide_kernel<1, true, true> : migrate_wide_kernel<1, false, true>;
        else if (flags & IMG2D_FLAG_WIDE_SCALAR)
            wf = stage ? migrate_wide_kernel<0, true> : migrate_wide_kernel<0, false>;
        else if (cluster2_mp(M) > 64)
            return false;  // a warp's 64 positions cover the operator's reach at every length that fits
        else
            wf = stage ? migrate_wide_kernel<1, true, false, 4, true> : migrate_wide_kernel<1, false, false, 4, true>;
        const size_t smemw = (stage ? wide_stage_smem_bytes(M) : wide_smem_bytes(M)) + bars;
        if (smemw + static_reserve > (size_t)smem_optin) return false;
        int widest = make_groups(WideShape::G);
        int K = (widest + WideShape::PC - 1) / WideShape::PC;
        p->packing = "lines";
        p->pack_cost = 0.0;
        for (const GroupDesc &g : groups) p->pack_cost += wide_item_cost(g.W, K);
        if (!(flags & IMG2D_FLAG_LINE_PACKING) && p->ns <= kWindowPackingMaxShots) {
            // window-first packing where it costs at least 1% less, on clusters just wide enough for
            // the widest shot or one CTA wider (wider windows chain more shots per lane slot);
            // cluster sizes beyond the portable 8 only where the line packing needs them anyway
            const int Kw = (*std::max_element(p->w.begin(), p->w.end()) + WideShape::PC - 1) / WideShape::PC;
            const int Kline = K;
            for (int Kc = Kw; Kc <= Kw + 1; ++Kc) {
                if (Kc > 8 && Kc != Kline) continue;
                std::vector<GroupDesc> g2;
                std::vector<int4> s2;
                std::vector<int16_t> o2;
                const double cost2 = pack_windows_best(p, WideShape::G, Kc, g2, s2, o2);
                if (cost2 > 0.0 && cost2 < p->pack_cost * 0.99) {
                    groups.swap(g2);
                    segs.swap(s2);
                    owner.swap(o2);
                    K = Kc;
                    widest = 0;
                    for (const GroupDesc &g : groups) widest = std::max(widest, g.W);
                    p->packing = "windows";
                    p->pack_cost = cost2;
                }
            }
        }
        if (!(K <= 8 || (K <= kMaxCluster && clusters_that_fit((const void *)wf, K, WideShape::NW * 32, smemw) > 0)))
            return false;
        p->cluster = K;
        p->G = WideShape::G;
        p->fixed = true;
        p->fn = wf;
        p->smem = smemw;
        p->max_w = widest;
        p->block = WideShape::NW * 32;
        p->variant = ((flags & IMG2D_FLAG_WIDE_SCALAR) ? 0 : 1) + (stage ? 2 : 0) + (bulk ? 4 : 0);
        p->kname = "migrate_wide";
        return true;
    };
    const int wide_flags = IMG2D_FLAG_WIDE | IMG2D_FLAG_WIDE_SCALAR | IMG2D_FLAG_WIDE_BULK;
    if ((flags & IMG2D_FLAG_WIDE_BULK) && (flags & IMG2D_FLAG_WIDE_SCALAR))
        return fail(IMG2D_EINVAL, "IMG2D_FLAG_WIDE_BULK runs packed FMAs; it does not combine with "
                                  "IMG2D_FLAG_WIDE_SCALAR");
    const bool wide_requested = (flags & wide_flags) != 0;
    const bool explicit_kernel = wide_requested || explicit_variant || tab16 ||
                                 (flags & (IMG2D_FLAG_GENERIC | IMG2D_FLAG_NO_CLUSTER | IMG2D_FLAG_CLUSTER_V1 |
                                           IMG2D_FLAG_CLUSTER2 | IMG2D_FLAG_LINE_PACKING)) != 0;
    const bool wide_ok = mode == OP_CONJ && !tab16 && p->L >= 7 &&
                         !(flags & (IMG2D_FLAG_GENERIC | IMG2D_FLAG_NO_CLUSTER | IMG2D_FLAG_CLUSTER_V1 |
                                    IMG2D_FLAG_CLUSTER2)) &&
                         !explicit_variant && (wide_requested || p->n_slots >= 6);
    bool want_wide = wide_ok && wide_requested;
    if (wide_ok && !wide_requested) {
        // default choice: SMs the cluster2 kernel would keep busy on this geometry
        const int pc2 = cv.nw * 32;
        const size_t smem2 = cluster2_smem_bytes(M, pc2) + (cv.stage ? cluster2_stage_bytes(pc2) : 0) +
                             (cv.ring ? cluster2_ring_bytes(pc2) : 0);
        const int K2 = (make_groups(16) + pc2 - 1) / pc2;
        const int busy = smem2 + static_reserve <= (size_t)smem_optin && K2 <= kMaxCluster
                             ? clusters_that_fit((const void *)cv.fn, K2, pc2, smem2) * K2
                             : 0;
        want_wide = p->n_slots < 12 || busy < nsm * 96 / 100;
    }
    // The row-split kernel instead: always for a table pair and for fewer than 6 slots, else where either of
    // two estimates finds it faster than the kernel chosen below.  Its results are the nearer ones to 64
    // bits (four short sums per output in place of a long one: 2.6e-7 and 5.3e-7 on the gradient of 168
    // ragged shots, 35 taps), so one of the two is enough.  Surveys of 12 slots or more are only
    // considered when its items fill the SMs (the estimates are made for that).
    int rows_G = 1;
    std::vector<int> rows_W;  // its items' windows
    // Its CTAs have a partial image and compensation each.  Those of several CTAs per SM take at most 8 GB:
    // 5 shots of 600 traces over 4096 x 1000, 256 frequencies, took 14.5 GB.
    const int rows_most = (int)std::max<size_t>(1, (8ull << 30) / ((size_t)nsm * nextrap * nx * 8));
    RowsLaunch rows_l{1, 1e30};
    int rows_smem_sm = 0;
    if (mode != OP_DENSE && !explicit_kernel && find_rows(1, p->L, mode == OP_TWO)) {
        IMG2D_CUDA(cudaDeviceGetAttribute(&rows_smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
        for (int G = 1; G <= std::min(2, p->n_slots); ++G) {
            const int widest = make_groups(G);
            if (rows_smem_bytes(G, widest, p->L) + static_reserve > (size_t)smem_optin) continue;
            const long long n = (long long)groups.size() * nf;
            if (p->n_slots >= 12 && mode == OP_CONJ && n < nsm) continue;
            const RowsLaunch r = rows_launch(G, widest, p->L, mode == OP_TWO, n, nsm, rows_smem_sm, rows_most);
            if (r.us < rows_l.us) {
                rows_l = r;
                rows_G = G;
                rows_W.clear();
                for (const GroupDesc &g : groups) rows_W.push_back(g.W);
            }
        }
        if (rows_l.us < 1e30) {
            if (mode == OP_TWO || p->n_slots < 6) {
                p->rows = true;
            } else {
                // By waves of the widest window of a line packing.  Time of a depth step of the wide kernel (8
                // slots x up to 1024 positions per CTA) or of the 16-slot one (up to 512), in
                // microseconds, for a CTA with all warps busy.  Clusters of three and more leave about
                // 9% of the SMs idle.
                const bool wide = want_wide;
                const int G = wide ? WideShape::G : 16, pc = wide ? WideShape::PC : 512;
                const int widest = make_groups(G), K = (widest + pc - 1) / pc;
                const int nc = std::min(pc, (widest + K * 256 - 1) / (K * 256) * 256);
                const double item = wide ? 0.344 * (p->L + 15) * wide_item_cost(nc, 1)
                                         : 0.375 * (p->L + 7.4) * (nc == pc ? 1.0 : 0.57);
                const int clusters = std::max(1, (K > 2 ? nsm * 91 / 100 : nsm) / K);
                const double waves = (double)groups.size() * nf / clusters;
                p->rows = 1.08 * rows_l.us < item * (waves <= 4.0 ? std::ceil(waves) : waves + 0.5);
            }
        }
    }
    // The 16-slot default: the wide kernel's step with 8 lanes per group (16 slots x 512 positions per
    // CTA, clusters as cluster2's), reported as the cluster2 variant after those of the table.
    auto try_wide16 = [&]() {
        const bool stage = wide_stage_smem_bytes<Wide16Shape>(M) + static_reserve <= (size_t)smem_optin;
        const size_t smemw = stage ? wide_stage_smem_bytes<Wide16Shape>(M) : wide_smem_bytes<Wide16Shape>(M);
        if (smemw + static_reserve > (size_t)smem_optin) return false;
        // up to 65 taps a warp's 32 positions cover the operator's reach: waits for neighbours only
        if (cluster2_mp(M) > 32) return false;
        KernelFn wf = stage ? migrate_wide_kernel<1, true, false, 8, true> : migrate_wide_kernel<1, false, false, 8, true>;
        const int widest = make_groups(Wide16Shape::G);
        const int K = (widest + Wide16Shape::PC - 1) / Wide16Shape::PC;
        if (!(K <= 8 || (K <= kMaxCluster && clusters_that_fit((const void *)wf, K, Wide16Shape::NW * 32, smemw) > 0)))
            return false;
        p->cluster = K;
        p->G = Wide16Shape::G;
        p->fixed = true;
        p->fn = wf;
        p->smem = smemw;
        p->max_w = widest;
        p->block = Wide16Shape::NW * 32;
        p->variant = kNumCluster2 + (stage ? 0 : 1);
        p->kname = "migrate_cluster2";
        return true;
    };
    if (!p->rows && want_wide) try_wide();
    if (!p->cluster && !p->rows && cluster_ok && !explicit_kernel && p->L >= 7) try_wide16();
    if (!p->cluster && !p->rows && cluster_ok && !(flags & (IMG2D_FLAG_CLUSTER_V1 | wide_flags)) &&
        p->L >= 7) {
        // the default ring variant needs 33 KB more shared memory than the staged one: long
        // operators or very wide windows fall back to the staged variant
        if (!try_cluster2(cv, vsel) && !explicit_variant && !tab16 && vsel != kCluster2Staged)
            try_cluster2(kCluster2[kCluster2Staged], kCluster2Staged);
    }
    if (tab16 && !p->cluster)
        return fail(IMG2D_EINVAL, "16-bit operator tables need the cluster kernel (>= 12 lane slots, 2M+1 >= 7, "
                                  "window <= 16 CTAs)");
    p->tab16 = tab16;
    const ClusterKernel *ck = cluster_ok ? find_cluster(p->L) : nullptr;
    if (!p->cluster && !p->rows && ck && ck->smem + static_reserve <= (size_t)smem_optin) {
        const int widest = make_groups(ClusterShape::G);
        const int K = (widest + ClusterShape::PC - 1) / ClusterShape::PC;
        if (K <= 8) {
            p->cluster = K == 1 ? 1 : (K <= 2 ? 2 : (K <= 4 ? 4 : 8));
            p->G = ClusterShape::G;
            p->fixed = true;
            p->fn = ck->fn;
            p->smem = ck->smem;
            p->max_w = widest;
            p->kname = "migrate_cluster";
        }
    }
    if (!p->rows && rows_l.us < 1e30 && !p->cluster) p->rows = true;  // a lane per output: two to six times slower
    if (!p->rows && rows_l.us < 1e30 && nf >= 16) {
        // Either kernel's items, widest first, through the queue of its CTAs or clusters.  Microseconds per
        // depth step and item, fitted on a B200 to 316 surveys of 6 to 256 shots, 16 to 256 frequencies,
        // 100 to 4096 positions, 19 to 55 taps: the wide kernel (8 slots) and the 16-slot one within 4%
        // (standard deviation), the row-split one within 5 (a slot) and 6.5% (two), which is the margin.
        // 8 of the surveys take the row-split kernel by this estimate only, 3 to 27% faster.
        const size_t rsmem = rows_smem_bytes(rows_G, *std::max_element(rows_W.begin(), rows_W.end()), p->L) + 1024;
        const int per_sm = (int)std::min<size_t>(16 / rows_l.warps, rows_smem_sm / rsmem);  // 128 registers a thread
        const int slots = (int)std::min<long long>((long long)rows_W.size() * nf, (long long)nsm * std::max(std::min(per_sm, rows_most), 1));
        const int per = (slots + nsm - 1) / nsm;  // CTAs that share an SM
        const int q = rows_np(p->L);
        // 3 pairs of taps cost as much as 4: their second chunk of 2 taps is a load of its own
        const double round = rows_G == 1 ? 0.11 + 0.0615 * q
                                         : (0.123 + 0.103 * (q == 3 ? 4 : q)) * std::pow(plan_row_starts(p).passes, 0.117) *
                                               (per > 1 ? 0.905 : 1.0);
        std::vector<double> mine, other;
        for (int W : rows_W) {
            const int nwb = (W + kRowsWarpPos - 1) / kRowsWarpPos;
            const int rounds = (nwb + rows_l.warps - 1) / rows_l.warps;
            const double active = (double)per * nwb / rounds;  // warps on the SM
            mine.push_back(round * (rounds * (1.0 + 0.25 * active) + (rows_G == 1 ? 1.0 : 0.6)));
        }
        const bool wide = p->G == WideShape::G;
        const int pc = wide ? WideShape::PC : 512, K = p->cluster;
        for (const GroupDesc &g : groups) {
            const double share = (double)std::min(pc, (g.W + K * 256 - 1) / (K * 256) * 256) / pc;
            other.push_back(wide ? 1.4 + 0.083 * p->L + (4.7 + 0.25 * p->L) * share
                                 : 1.5 + 0.02 * p->L + (0.85 + 0.35 * p->L) * share);
        }
        const int clusters = std::max(1, clusters_that_fit((const void *)p->fn, K, p->block, p->smem));
        p->rows = 1.06 * queue_time(mine, nf, slots) < queue_time(other, nf, clusters);
    }
    if (p->rows) {
        p->cluster = 0;
        p->variant = -1;
        p->packing = "lines";
        p->pack_cost = 0.0;
        p->G = rows_G;
        p->fixed = true;
        p->fn = find_rows(rows_G, p->L, mode == OP_TWO);
        p->max_w = make_groups(rows_G);
        p->smem = rows_smem_bytes(rows_G, p->max_w, p->L);
        p->block = 32 * rows_l.warps;
        p->kname = "migrate_rows";
    }
    if (!p->cluster && !p->rows) {
        int nsp2 = 1;
        while (nsp2 < p->n_slots) nsp2 <<= 1;
        int G = 8;
        while (G > 1 && (G > nsp2 || smem_bytes(G, nx, M, kX) + static_reserve > (size_t)smem_optin)) G >>= 1;
        const bool use_fixed = (mode == OP_CONJ) && !(flags & IMG2D_FLAG_GENERIC) && find_fixed(G, p->L);
        const int X = use_fixed ? kX : 4;
        if (smem_bytes(G, nx, M, X) + static_reserve > (size_t)smem_optin)
            return fail(IMG2D_EINVAL, "aperture too wide for one CTA's shared memory");
        p->G = G;
        p->fixed = use_fixed;
        p->fn = use_fixed ? find_fixed(G, p->L) : find_generic(G, mode);
        p->max_w = make_groups(G);
        p->smem = smem_bytes(G, p->max_w, M, X);
        p->kname = use_fixed ? "migrate_fixed" : "migrate_generic";
    }
    // Items (group, frequency), widest groups first so the tail of the queue is short work.
    std::vector<int2> items;
    items.reserve(groups.size() * (size_t)nf);
    std::vector<int> gorder(groups.size());
    std::iota(gorder.begin(), gorder.end(), 0);
    std::stable_sort(gorder.begin(), gorder.end(), [&](int a, int b) { return groups[a].W > groups[b].W; });
    for (int g : gorder)
        for (int j = 0; j < nf; ++j) items.push_back(make_int2(g, j));
    p->n_items = (int)items.size();
    p->group_order = gorder;
    {
        // (slot, position) pairs the kernel computes per depth step and frequency, per useful one
        double computed = 0.0, useful = 0.0;
        for (int s = 0; s < ns; ++s) useful += p->w[s];
        const int K = std::max(1, p->cluster);
        for (const GroupDesc &g : groups) {
            if (!strcmp(p->kname, "migrate_wide"))
                computed += (double)K * std::min(WideShape::PC, (g.W + K * 256 - 1) / (K * 256) * 256) * p->G;
            else if (!strcmp(p->kname, "migrate_cluster2"))
                computed += (double)K * p->block * p->G;
            else
                computed += (double)g.W * p->G;
        }
        p->computed_per_useful = computed / useful;
    }
    IMG2D_CUDA(cudaFuncSetAttribute(p->fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p->smem));
    if (p->cluster) {
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = p->cluster;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.gridDim = dim3(p->cluster * 64, 1, 1);
        cfg.blockDim = dim3(p->block, 1, 1);
        cfg.dynamicSmemBytes = p->smem;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int nclusters = 0;
        IMG2D_CUDA(cudaOccupancyMaxActiveClusters(&nclusters, (void *)p->fn, &cfg));
        if (nclusters <= 0) return fail(IMG2D_ECUDA, "no cluster of this size fits on the device");
        p->grid = std::min(p->n_items, nclusters) * p->cluster;
    } else if (p->rows) {
        int per_sm = 0;
        IMG2D_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, p->fn, p->block, p->smem));
        if (per_sm <= 0) return fail(IMG2D_ECUDA, "the row-split kernel does not fit on an SM");
        p->grid = std::min(p->n_items, nsm * std::min(per_sm, rows_most));
    } else {
        p->grid = std::min(p->n_items, nsm);
    }

    int rc;
    const size_t plane = (size_t)nextrap * nx;
    const size_t rows_tab_b = p->rows ? (size_t)nk * rows_row_floats(p->L, mode == OP_TWO) * sizeof(float) : 0;
    if ((rc = p->items.ensure(items.size() * sizeof(int2)))) return rc;
    if ((rc = p->groups.ensure(groups.size() * sizeof(GroupDesc)))) return rc;
    if ((rc = p->segs.ensure(segs.size() * sizeof(int4)))) return rc;
    if ((rc = p->owner.ensure(owner.size() * sizeof(int16_t)))) return rc;
    if ((rc = p->shot_off.ensure(p->off.size() * sizeof(long long)))) return rc;
    if ((rc = p->counter.ensure(2 * sizeof(int)))) return rc;  // work-queue counter, status word
    if (p->carver) {
        // ordered on the caller's stream after any earlier call that used the same scratch
        cudaStream_t us = p->upload_stream;
        IMG2D_CUDA(cudaMemcpyAsync(p->items.p, items.data(), items.size() * sizeof(int2), cudaMemcpyHostToDevice, us));
        IMG2D_CUDA(cudaMemcpyAsync(p->groups.p, groups.data(), groups.size() * sizeof(GroupDesc), cudaMemcpyHostToDevice, us));
        IMG2D_CUDA(cudaMemcpyAsync(p->segs.p, segs.data(), segs.size() * sizeof(int4), cudaMemcpyHostToDevice, us));
        IMG2D_CUDA(cudaMemcpyAsync(p->owner.p, owner.data(), owner.size() * sizeof(int16_t), cudaMemcpyHostToDevice, us));
        IMG2D_CUDA(cudaMemcpyAsync(p->shot_off.p, p->off.data(), p->off.size() * sizeof(long long), cudaMemcpyHostToDevice, us));
        IMG2D_CUDA(cudaMemsetAsync(p->counter.p, 0, 2 * sizeof(int), us));
        // pageable sources: make sure the copies have read the host vectors before they go away
        IMG2D_CUDA(cudaStreamSynchronize(us));
    } else {
        IMG2D_CUDA(cudaMemcpy(p->items.p, items.data(), items.size() * sizeof(int2), cudaMemcpyHostToDevice));
        IMG2D_CUDA(cudaMemcpy(p->groups.p, groups.data(), groups.size() * sizeof(GroupDesc), cudaMemcpyHostToDevice));
        IMG2D_CUDA(cudaMemcpy(p->segs.p, segs.data(), segs.size() * sizeof(int4), cudaMemcpyHostToDevice));
        IMG2D_CUDA(cudaMemcpy(p->owner.p, owner.data(), owner.size() * sizeof(int16_t), cudaMemcpyHostToDevice));
        IMG2D_CUDA(cudaMemcpy(p->shot_off.p, p->off.data(), p->off.size() * sizeof(long long), cudaMemcpyHostToDevice));
        const int zero[2] = {0, 0};  // (a copy: complete on return, whatever stream the plan is used on)
        IMG2D_CUDA(cudaMemcpy(p->counter.p, zero, sizeof(zero), cudaMemcpyHostToDevice));
    }
    if (p->carver) {
        // fixed scratch: fewer persistent CTAs when their private image partials would not fit
        const size_t idx_b = (size_t)nf * nextrap * ((nx + 7) / 8 * 8) * sizeof(uint16_t) + 256;
        const size_t tab_b = ((size_t)nk * ((p->L + 1) / 2 * 2) * sizeof(cpx) + 256) * (mode == OP_TWO ? 2 : 1);
        const size_t used = (p->carver->used + 255) & ~(size_t)255;
        const size_t left = p->carver->cap > used + idx_b + tab_b ? p->carver->cap - used - idx_b - tab_b : 0;
        const size_t fit = left / (2 * plane * sizeof(float) + 512);
        if (fit < 1)
            return fail(IMG2D_EINVAL, "problem needs more than the " + std::to_string(p->carver->cap >> 20) +
                                          " MiB of fixed scratch of the no-allocation entry point");
        p->grid = (int)std::min<size_t>((size_t)p->grid, fit);
    }
    while (mode != OP_DENSE) {  // dense calls take the images of the single shots only
        rc = p->partial.ensure((size_t)p->grid * plane * sizeof(float));
        if (!rc && (!p->rows || p->n_items > p->grid))  // one item per CTA needs no compensation
            rc = p->comp.ensure((size_t)p->grid * plane * sizeof(float));
        if (!rc) break;
        // the row-split kernel has several CTAs per SM: with less memory it runs on fewer
        if (rc != IMG2D_ENOMEM || !p->rows || p->grid <= 1) return rc;
        p->partial.release();
        p->grid = p->grid > nsm ? std::max(nsm, p->grid / 2) : p->grid / 2;
    }
    if (mode != OP_DENSE) {
        p->idx_lstride = (nx + 7) / 8 * 8;
        if ((rc = p->idx.ensure((size_t)nf * nextrap * p->idx_lstride * sizeof(uint16_t)))) return rc;
        p->tab_stride = (p->L + 1) / 2 * 2;
        if ((rc = p->tabF.ensure((size_t)nk * p->tab_stride * sizeof(cpx)))) return rc;
        if (p->tab16 && (rc = p->tab16buf.ensure((size_t)nk * p->tab_stride * sizeof(unsigned)))) return rc;
        if (mode == OP_TWO && (rc = p->tabB.ensure((size_t)nk * p->tab_stride * sizeof(cpx)))) return rc;
    }
    if (p->rows) {
        if ((rc = p->visits.ensure((size_t)p->grid * sizeof(int)))) return rc;
        if ((rc = p->tab_rows.ensure(rows_tab_b))) return rc;
    }
    return IMG2D_OK;
}

static MigrateArgs base_args(img2d_plan *p, cpx *wave, cpx *shot)
{
    MigrateArgs a{};
    a.nextrap = p->nextrap;
    a.nx = p->nx;
    a.nf = p->nf;
    a.M = p->M;
    a.tab_stride = p->tab_stride;
    a.n_items = p->n_items;
    a.items = p->items.as<int2>();
    a.groups = p->groups.as<GroupDesc>();
    a.segs = p->segs.as<int4>();
    a.owner = p->owner.as<int16_t>();
    a.shot_off = p->shot_off.as<long long>();
    a.tabF = p->tabF.as<cpx>();
    a.tabB = p->mode == OP_TWO ? p->tabB.as<cpx>() : p->tabF.as<cpx>();
    a.tab16 = p->tab16buf.p;
    if (p->rows) {
        a.tab_rows = p->tab_rows.p;
        const RowsStarts &rs = plan_row_starts(p);
        for (int i = 0; i < 4; ++i) a.row_start[i] = rs.s[i];
        a.row_apart = rs.apart;
    }
    a.idx = p->idx.as<uint16_t>();
    a.idx_jstride = (long long)p->nextrap * p->idx_lstride;
    a.idx_lstride = p->idx_lstride;
    a.wave = wave;
    a.shot = shot;
    a.write_back = 1;
    a.counter = p->counter.as<int>();
    return a;
}

// Status word (after the work-queue counter), read on `st`.  Launches only ever set it: it keeps the
// failure of any launch since the last reading, which clears it.
static int read_status(img2d_plan *p, cudaStream_t st)
{
    int status = 0;
    IMG2D_CUDA(cudaMemcpyAsync(&status, p->counter.as<int>() + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
    IMG2D_CUDA(cudaStreamSynchronize(st));
    if (status) {
        IMG2D_CUDA(cudaMemsetAsync(p->counter.as<int>() + 1, 0, sizeof(int), st));
        return fail(IMG2D_ECUDA, "a bounded wait inside a kernel of this plan gave up (status " + std::to_string(status) +
                                     "): results since the last status check are not valid");
    }
    return IMG2D_OK;
}

// The plan's persistent migration kernel on `grid` CTAs (whole clusters) of stream st.
static int launch_kernel(img2d_plan *p, const MigrateArgs &a, int grid, cudaStream_t st)
{
    if (p->cluster) {
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = p->cluster;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.gridDim = dim3(grid, 1, 1);
        cfg.blockDim = dim3(p->block, 1, 1);
        cfg.dynamicSmemBytes = p->smem;
        cfg.stream = st;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        IMG2D_CUDA(cudaLaunchKernelEx(&cfg, p->fn, a));
    } else {
        p->fn<<<grid, p->block, p->smem, st>>>(a);
    }
    IMG2D_CUDA(cudaGetLastError());
    return IMG2D_OK;
}

// Launch the persistent kernel and (optionally) reduce the stacked image.
static int launch(img2d_plan *p, MigrateArgs a, float *d_image, float *d_image_shots,
                  long long img_sstride, cudaStream_t st)
{
    const size_t plane = (size_t)p->nextrap * p->nx;
    IMG2D_CUDA(cudaMemsetAsync(p->counter.p, 0, sizeof(int), st));
    a.status = p->counter.as<int>() + 1;
    p->launched = true;
    if (d_image && p->rows) {
        IMG2D_CUDA(cudaMemsetAsync(p->visits.p, 0, (size_t)p->grid * sizeof(int), st));
        a.partial = p->partial.as<float>();
        a.comp = p->comp.as<float>();
        a.visits = p->visits.as<int>();
    } else if (d_image) {
        IMG2D_CUDA(cudaMemsetAsync(p->partial.p, 0, (size_t)p->grid * plane * sizeof(float), st));
        IMG2D_CUDA(cudaMemsetAsync(p->comp.p, 0, (size_t)p->grid * plane * sizeof(float), st));
        a.partial = p->partial.as<float>();
        a.comp = p->comp.as<float>();
    }
    if (d_image_shots) {
        IMG2D_CUDA(cudaMemset2DAsync(d_image_shots, img_sstride * sizeof(float), 0, plane * sizeof(float),
                                     p->ns, st));
        a.image_shots = d_image_shots;
        a.img_sstride = img_sstride;
    }
    if (p->timing && !p->ev0) {
        IMG2D_CUDA(cudaEventCreate(&p->ev0));
        IMG2D_CUDA(cudaEventCreate(&p->ev1));
    }
    if (p->timing) IMG2D_CUDA(cudaEventRecord(p->ev0, st));
    int rc;
    if ((rc = launch_kernel(p, a, p->grid, st))) return rc;
    if (p->timing) {
        IMG2D_CUDA(cudaEventRecord(p->ev1, st));
        p->ev_recorded = true;
    }
    if (d_image) {
        const int blocks = (int)std::min<size_t>((plane + 31) / 32, 148 * 64);
        reduce_partials_kernel<<<blocks, 256, 0, st>>>(p->partial.as<float>(), p->comp.as<float>(), a.visits, p->grid,
                                                       (long long)plane, d_image);
        IMG2D_CUDA(cudaGetLastError());
    }
    return IMG2D_OK;
}

// The row-split kernels' copy of the plan's tables.  Made by set_model where migration uses it, and by the
// first demigration that does; from then on every set_model renews it, so that a captured call,
// which holds the address and not the copying, reads the model of the last set_model.
static size_t rows_table_bytes(const img2d_plan *p)
{
    return (size_t)p->nk * rows_row_floats(p->L, p->mode == OP_TWO) * sizeof(float);
}
static int set_rows_table(img2d_plan *p, cudaStream_t st)
{
    const bool two = p->mode == OP_TWO;
    const long long floats = (long long)(rows_table_bytes(p) / sizeof(float));
    const int rc = p->tab_rows.ensure(rows_table_bytes(p));
    if (rc) return rc;
    rows_table_kernel<<<(int)std::min<long long>((floats / 2 + 255) / 256, 148 * 8), 256, 0, st>>>(
        p->tabF.as<cpx>(), two ? p->tabB.as<cpx>() : nullptr, p->tab_stride, p->L, rows_np(p->L), plan_row_starts(p),
        p->nk, p->tab_rows.as<float>());
    IMG2D_CUDA(cudaGetLastError());
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &capture) != cudaSuccess) cudaGetLastError();
    if (capture == cudaStreamCaptureStatusNone) p->rows_tab_set = true;  // a captured copy has not run yet
    return IMG2D_OK;
}

static int set_model(img2d_plan *p, const double *d_omega, const double *d_vel, double dk,
                     const cpx *d_tabF, const cpx *d_tabB, cudaStream_t st)
{
    p->adj_cache_valid = false;
    if (!d_omega || !d_vel || !d_tabF || !(dk > 0.0))
        return fail(IMG2D_EINVAL, "set_model needs omega, velocity, tab_forw and dk > 0");
    if (p->mode == OP_TWO && !d_tabB) return fail(IMG2D_EINVAL, "two-table mode needs tab_back");
    const size_t row = (size_t)p->L * sizeof(cpx), prow = (size_t)p->tab_stride * sizeof(cpx);
    IMG2D_CUDA(cudaMemsetAsync(p->tabF.p, 0, (size_t)p->nk * prow, st));
    IMG2D_CUDA(cudaMemcpy2DAsync(p->tabF.p, prow, d_tabF, row, row, p->nk, cudaMemcpyDeviceToDevice, st));
    if (p->mode == OP_TWO) {
        IMG2D_CUDA(cudaMemsetAsync(p->tabB.p, 0, (size_t)p->nk * prow, st));
        IMG2D_CUDA(cudaMemcpy2DAsync(p->tabB.p, prow, d_tabB, row, row, p->nk, cudaMemcpyDeviceToDevice, st));
    }
    if (p->rows || p->tab_rows.p) {
        const int rc = set_rows_table(p, st);
        if (rc) return rc;
    }
    if (p->tab16) {
        const long long n = (long long)p->nk * p->tab_stride;
        table_to_16bit_kernel<<<(int)std::min<long long>((n + 255) / 256, 148 * 8), 256, 0, st>>>(
            p->tabF.as<cpx>(), n, p->tab16 == 2, p->tab16buf.as<unsigned>());
        IMG2D_CUDA(cudaGetLastError());
    }
    const long long total = (long long)p->nf * p->nextrap * p->nx;
    const int blocks = (int)std::min<long long>((total + 255) / 256, 148 * 16);
    index_table_kernel<<<blocks, 256, 0, st>>>(d_omega, d_vel, p->nf, p->nextrap, p->nx, p->idx_lstride, p->nk,
                                               dk, p->idx.as<uint16_t>());
    IMG2D_CUDA(cudaGetLastError());
    p->model_set = true;
    return IMG2D_OK;
}

// Row-split demigration: the kept source of all items takes at most this many complex values (8 GB);
// above, IMG2D_SOURCE_KEEP keeps nothing of use and every call steps the source again, which costs
// what the slab recomputation from kept checkpoints costs the other kernels.
constexpr long long kDemigRowsCacheElems = 1ll << 30;

// Launch state of the demigration: its own slot groups (one complex wavefield per slot, so up to
// 8 slots fit beside the halos), items, and the per-CTA checkpoint / slab / save planes.
static int demig_prepare(img2d_plan *p, int slab)
{
    if (slab <= 0) slab = 8;
    slab = std::min(slab, p->nextrap);
    const int nslab = (p->nextrap + slab - 1) / slab;
    if ((p->adj_fn || p->adj_rows_fn || p->adj_wide_fn) && p->adj_slab == slab) return IMG2D_OK;
    p->adj_cache_valid = false;  // the checkpoint layout depends on the slab depth
    int dev = 0, smem_optin = 0, nsm = 0;
    IMG2D_CUDA(cudaGetDevice(&dev));
    IMG2D_CUDA(cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    IMG2D_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const int static_reserve = 1024;
    std::vector<GroupDesc> groups;
    std::vector<int4> segs;
    std::vector<int16_t> owner;
    int G = 8, widest = 0, K = 0;
    bool ring = false;
    DemigFn fn = nullptr;
    size_t smem = 0;
    // With enough slots to fill items of 16: the wide kernel (up to 1024 positions per CTA; 7 to 65 taps) or
    // the cluster kernel (512 positions, any length), where the widest window fits 16 CTAs; otherwise
    // the row-split kernel or the single-CTA one.
    //
    // The wide kernel's windows may be spread over more CTAs than they need, and the cluster kernel has
    // unrolled instances for 25, 31 and 35 taps.  Both are chosen by the time of their items through the
    // queue, in microseconds per depth step of a call that recomputes its source (within 6% of 110
    // calls on a B200, 12 to 189 shots of 100 to 3300 positions; the cluster kernel at run-time
    // lengths takes 1.5 to 5 times as long; in clusters less than 512 positions a CTA are no faster).  A lane of the wide kernel has four slots and a warp twice
    // the positions, so windows of 400 to 512 leave it half its warps: 13 shots of 437, 170 frequencies,
    // 35 taps 3.03 ms, the cluster kernel 2.91.
    void (*wide_fn)(DemigrateArgs, int *) = nullptr;
    const bool slots16 = p->n_slots >= 12 && !(p->flags & IMG2D_FLAG_NO_CLUSTER);
    const DemigFn ring_fn = slots16 && !(p->flags & IMG2D_FLAG_DEMIG_NO_RING) ? find_demig_cluster(p->L) : nullptr;
    auto cluster_fits = [&](DemigFn f, int k, size_t bytes) {
        return f && bytes + static_reserve <= (size_t)smem_optin &&
               (k <= 8 || (k <= kMaxCluster && clusters_that_fit((const void *)f, k, kDcNW * 32, bytes) > 0));
    };
    if (p->adj_allow_wide && slots16 && p->L >= 7 && demigw_smem_bytes(p->M) + static_reserve <= (size_t)smem_optin) {
        widest = pack_groups(p, DemigWideShape::G, groups, segs, owner);
        // operators of less than 17 taps need few pairs per step: the wait for the ring's first copies
        // would be most of it
        const bool wring = !(p->flags & IMG2D_FLAG_DEMIG_NO_RING) && p->L >= 17;
        auto wf = wring ? demigrate_wide_kernel<true> : demigrate_wide_kernel<false>;
        const size_t wsmem = demigw_smem_bytes(p->M);
        const int least = (widest + DemigWideShape::PC - 1) / DemigWideShape::PC;
        double best = 1e30;
        for (int k = least; k == least || (k <= 8 && widest / k >= 256); ++k) {
            // (no more planes than 512 positions per CTA would have)
            if (k > least && k * demigw_share(widest, k) > (widest + 511) / 512 * 512) continue;
            const int n = k <= kMaxCluster ? clusters_that_fit((const void *)wf, k, DemigWideShape::NW * 32, wsmem) : 0;
            if (n <= 0) continue;
            std::vector<double> cost;
            for (const GroupDesc &g : groups)
                cost.push_back(10.2 + (k > 1 ? 0.52 : 0.43) * p->L +
                               (0.0045 + 0.00066 * p->L) * std::max(k > 1 ? 512 : 0, demigw_share(g.W, k)));
            const double t = queue_time(cost, p->nf, n);
            if (t < best) {
                best = t;
                K = k;
            }
        }
        const int kc = (widest + kDcPC - 1) / kDcPC;
        const size_t csmem = demigc_ring_smem_bytes(p->M);
        if (K && cluster_fits(ring_fn, kc, csmem)) {
            const std::vector<double> cost(groups.size(), (kc > 1 ? 10.0 : 9.0) + 0.81 * p->L);
            const int n = clusters_that_fit((const void *)ring_fn, kc, kDcNW * 32, csmem);
            if (n > 0 && queue_time(cost, p->nf, n) < best) K = 0;
        }
        if (K) {
            G = DemigWideShape::G;
            wide_fn = wf;
            smem = wsmem;
            ring = wring;
        }
    }
    if (!K && slots16) {
        widest = pack_groups(p, 16, groups, segs, owner);
        const int k = (widest + kDcPC - 1) / kDcPC;
        for (DemigFn f : {ring_fn, (DemigFn)demigrate_cluster_kernel<0>}) {
            const size_t bytes = f == ring_fn ? demigc_ring_smem_bytes(p->M) : demigc_smem_bytes(p->M);
            if (K || !cluster_fits(f, k, bytes)) continue;
            K = k;
            G = 16;
            fn = f;
            smem = bytes;
            ring = f == ring_fn;
        }
    }
    // Fewer slots: the row-split kernel, which keeps every S_l, where its shared memory fits.
    void (*rows_fn)(RowsAdjArgs) = nullptr;
    if (!K && p->adj_allow_rows && p->n_slots < 12 && !(p->flags & (IMG2D_FLAG_NO_CLUSTER | IMG2D_FLAG_GENERIC))) {
        for (G = p->n_slots >= 2 ? 2 : 1; G >= 1 && !rows_fn; --G) {
            widest = pack_groups(p, G, groups, segs, owner);
            smem = rows_adj_smem_bytes(G, widest, p->L);
            if (smem + static_reserve <= (size_t)smem_optin) rows_fn = find_demig_rows(G, p->L);
        }
        G = rows_fn ? G + 1 : 8;
    }
    if (!K && !rows_fn) {
        for (;; G >>= 1) {
            widest = pack_groups(p, G, groups, segs, owner);
            if (demig_smem_bytes(G, widest, p->M) + static_reserve <= (size_t)smem_optin) break;
            if (G == 2) return fail(IMG2D_EINVAL, "aperture too wide for the demigration kernel's shared memory");
        }
        // fewer slots than lanes: smaller groups leave fewer idle lanes
        while (G > 2 && (int)p->slot_order.size() <= G / 2) G >>= 1;
        widest = pack_groups(p, G, groups, segs, owner);
        fn = find_demig(G, p->L);
        smem = demig_smem_bytes(G, widest, p->M);
    }
    if (!fn && !rows_fn && !wide_fn) return fail(IMG2D_EINVAL, "no demigration kernel for this configuration");
    const void *any_fn = rows_fn ? (const void *)rows_fn : (wide_fn ? (const void *)wide_fn : (const void *)fn);
    IMG2D_CUDA(cudaFuncSetAttribute(any_fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    std::vector<int2> items;
    std::vector<int> gorder(groups.size());
    std::iota(gorder.begin(), gorder.end(), 0);
    std::stable_sort(gorder.begin(), gorder.end(), [&](int a, int b) { return groups[a].W > groups[b].W; });
    for (int g : gorder)
        for (int j = 0; j < p->nf; ++j) items.push_back(make_int2(g, j));
    int grid = 0, block = kAdjWarps * 32;
    long long work_cta = 0;   // float2 elements of per-CTA work area
    long long cache_item = 0; // float2 elements of kept checkpoints per item
    if (K) {
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = K;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.gridDim = dim3(K * 64, 1, 1);
        cfg.blockDim = dim3(kDcNW * 32, 1, 1);
        cfg.dynamicSmemBytes = smem;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int nclusters = 0;
        IMG2D_CUDA(cudaOccupancyMaxActiveClusters(&nclusters, (void *)any_fn, &cfg));
        if (nclusters <= 0) return fail(IMG2D_ECUDA, "no demigration cluster of this size fits on the device");
        grid = (int)std::min<size_t>(items.size(), (size_t)nclusters) * K;
        // float4 per plane
        const long long pe4 = wide_fn ? (long long)demigw_share(widest, K) * DemigWideShape::ROW : (long long)kDcPC * kDcQ;
        work_cta = 2 * (long long)(nslab + slab + 1) * pe4;
        cache_item = 2 * (long long)K * nslab * pe4;
    } else if (rows_fn) {
        // warps: a forward step takes a round per 32 positions and warp, a transposed one (2.4 times
        // as long) per 64; the more warps share an SM the longer a round (rows_launch)
        int smem_sm = 0;
        IMG2D_CUDA(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
        const int wp = rows_adj_wp(widest), n64 = wp / kRowsAdjPos;
        const long long n_items = (long long)items.size();
        double best = 1e30;
        for (int w = 1; w <= std::min(n64, kRowsThreads / 32); ++w) {
            const long long c = std::min<long long>(16 / w, smem_sm / (long long)(smem + 1024));
            if (c < 1) continue;
            const double rounds = (2 * n64 + w - 1) / w + 2.4 * ((n64 + w - 1) / w);
            auto wave = [&](long long per_sm) { return rounds * (1.0 + per_sm * w / 6.0); };
            const long long full = n_items / (nsm * c), rest = n_items % (nsm * c);
            const double t = full * wave(c) + (rest ? wave((rest + nsm - 1) / nsm) : 0.0);
            if (t < best) {
                best = t;
                block = 32 * w;
            }
        }
        int bps = 0;
        IMG2D_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, any_fn, block, smem));
        if (bps <= 0) return fail(IMG2D_ECUDA, "the row-split demigration kernel does not fit on an SM");
        grid = (int)std::min<size_t>(items.size(), (size_t)nsm * bps);
        work_cta = (long long)p->nextrap * wp * G;
        cache_item = work_cta;
    } else {
        int bps = 0;
        IMG2D_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, fn, kAdjWarps * 32, smem));
        if (bps <= 0) return fail(IMG2D_ECUDA, "demigration kernel does not fit on an SM");
        grid = (int)std::min<size_t>(items.size(), (size_t)nsm * bps);
        work_cta = (long long)(nslab + slab + 1) * widest * G;
        cache_item = (long long)nslab * widest * G;
    }
    int rc;
    if ((rc = p->adj_items.ensure(items.size() * sizeof(int2)))) return rc;
    if ((rc = p->adj_groups.ensure(groups.size() * sizeof(GroupDesc)))) return rc;
    if ((rc = p->adj_segs.ensure(segs.size() * sizeof(int4)))) return rc;
    if ((rc = p->adj_owner.ensure(owner.size() * sizeof(int16_t)))) return rc;
    if ((rc = p->adj_counter.ensure(sizeof(int)))) return rc;
    if (!rows_fn && (rc = p->adj_work.ensure((size_t)grid * work_cta * sizeof(float2)))) {
        if (rc != IMG2D_ENOMEM || !wide_fn) return rc;
        p->adj_allow_wide = false;  // the cluster kernel's planes are half as large
        return demig_prepare(p, slab);
    }
    IMG2D_CUDA(cudaMemcpy(p->adj_items.p, items.data(), items.size() * sizeof(int2), cudaMemcpyHostToDevice));
    IMG2D_CUDA(cudaMemcpy(p->adj_groups.p, groups.data(), groups.size() * sizeof(GroupDesc), cudaMemcpyHostToDevice));
    IMG2D_CUDA(cudaMemcpy(p->adj_segs.p, segs.data(), segs.size() * sizeof(int4), cudaMemcpyHostToDevice));
    IMG2D_CUDA(cudaMemcpy(p->adj_owner.p, owner.data(), owner.size() * sizeof(int16_t), cudaMemcpyHostToDevice));
    p->adj_G = G;
    p->adj_grid = grid;
    p->adj_items_n = (int)items.size();
    p->adj_wmax = widest;
    p->adj_block = K ? kDcNW * 32 : block;
    p->adj_rows = rows_fn != nullptr;
    p->adj_wide_fn = wide_fn;
    p->adj_rows_fn = rows_fn;
    p->adj_full_cache = rows_fn && (long long)items.size() * cache_item <= kDemigRowsCacheElems;
    p->adj_cluster = K;
    p->adj_work_cta = work_cta;
    p->adj_cache_item = cache_item;
    p->adj_slab = slab;
    p->adj_nslab = nslab;
    p->adj_smem = smem;
    p->adj_fn = fn;
    p->adj_ring = ring;
    return IMG2D_OK;
}

// Scoped device allocation for the host entry points.
struct Scratch {
    struct Block {
        void *p;
        size_t bytes;
        int dev;
    };
    std::vector<Block> blocks;
    ~Scratch()
    {
        for (const Block &b : blocks) device_free(b.p, b.bytes, b.dev);
    }
    template <class T> int alloc(T **out, size_t n)
    {
        Block b{};
        const int rc = device_alloc(&b.p, n ? n : 16, &b.bytes, &b.dev);
        if (rc) return rc;
        blocks.push_back(b);
        *out = static_cast<T *>(b.p);
        return IMG2D_OK;
    }
};

// Dense-table drop-in: both argument orders come here.
// Sizes for which the reference's loops (cpp_src/extrapolation_cpu.cpp:39-99) do no extrapolation:
// ns, nx or nextrap zero leave every buffer as it was; nf zero writes zero image rows [0, nextrap).
// Handled on the host; returns 1 when the call is complete.
static int degenerate_call(int ns, int nextrap, int nz, int nx, int nf, float *image, int *rc)
{
    if (ns < 0 || nextrap < 0 || nz < 0 || nx < 0 || nf < 0 || nz < nextrap) {
        *rc = fail(IMG2D_EINVAL, "invalid dimensions (negative, or nz < nextrap)");
        return 1;
    }
    if (ns == 0 || nx == 0 || nextrap == 0) {
        *rc = IMG2D_OK;
        return 1;
    }
    if (nf == 0) {
        if (!image) {
            *rc = fail(IMG2D_EINVAL, "null image pointer");
            return 1;
        }
        for (int s = 0; s < ns; ++s)
            std::memset(image + (size_t)s * nz * nx, 0, (size_t)nextrap * nx * sizeof(float));
        *rc = IMG2D_OK;
        return 1;
    }
    return 0;
}

static int run_dense(int ns, int nextrap, int nz, int nx, int nf, int nt, int M, const cpx *opF,
                     const cpx *opB, cpx *wave, cpx *shot, float *image, int write_back)
{
    int rc;
    if (degenerate_call(ns, nextrap, nz, nx, nf, image, &rc)) return rc;
    if ((rc = check_device())) return rc;
    if (!opF || !opB || !wave || !shot || !image) return fail(IMG2D_EINVAL, "null pointer argument");
    img2d_plan plan;
    if ((rc = build_plan(&plan, ns, nextrap, nz, nx, nf, nt, M, 1, nullptr, nullptr, 0, OP_DENSE))) return rc;
    Scratch sc;
    const size_t L = 2 * (size_t)M + 1;
    const size_t tab = (size_t)nextrap * nf * nx * L;
    const size_t wel = (size_t)ns * nt * nx;
    const size_t plane = (size_t)nz * nx;
    cpx *dF, *dB, *dW, *dS;
    float *dI;
    if ((rc = sc.alloc(&dF, tab * sizeof(cpx)))) return rc;
    if ((rc = sc.alloc(&dB, tab * sizeof(cpx)))) return rc;
    if ((rc = sc.alloc(&dW, wel * sizeof(cpx)))) return rc;
    if ((rc = sc.alloc(&dS, wel * sizeof(cpx)))) return rc;
    if ((rc = sc.alloc(&dI, (size_t)ns * plane * sizeof(float)))) return rc;
    IMG2D_CUDA(cudaMemcpy(dW, wave, wel * sizeof(cpx), cudaMemcpyHostToDevice));
    IMG2D_CUDA(cudaMemcpy(dS, shot, wel * sizeof(cpx), cudaMemcpyHostToDevice));
    // The tables go up in up to eight slabs of depth steps (16 MB or more each), on a stream of their
    // own, while the kernel runs the slabs that have arrived (its wavefields pass from launch to launch
    // through dW and dS).
    const size_t depth = (size_t)nf * nx * L;  // table elements per depth step
    const int slabs = std::max(1, std::min(nextrap, (int)std::min<size_t>(8, tab * sizeof(cpx) >> 24)));
    auto first = [&](int c) { return (int)((long long)c * nextrap / slabs); };
    std::vector<UploadPiece> pieces;
    for (int c = 0; c < slabs; ++c) {
        const size_t at = first(c) * depth, n = (first(c + 1) - first(c)) * depth;
        add_pieces(pieces, dF + at, opF + at, n * sizeof(cpx), c);
        add_pieces(pieces, dB + at, opB + at, n * sizeof(cpx), c);
    }
    struct Queue {
        cudaStream_t s = nullptr;
        cudaEvent_t e = nullptr;
        ~Queue()
        {
            if (e) cudaEventDestroy(e);
            if (s) cudaStreamDestroy(s);
        }
    } up;
    IMG2D_CUDA(cudaStreamCreateWithFlags(&up.s, cudaStreamNonBlocking));
    IMG2D_CUDA(cudaEventCreateWithFlags(&up.e, cudaEventDisableTiming));
    IMG2D_CUDA(cudaMemset2DAsync(dI, plane * sizeof(float), 0, (size_t)nextrap * nx * sizeof(float), ns, 0));
    rc = upload(pieces, slabs, up.s, [&](int c) -> int {
        IMG2D_CUDA(cudaEventRecord(up.e, up.s));
        IMG2D_CUDA(cudaStreamWaitEvent(0, up.e, 0));
        MigrateArgs a = base_args(&plan, dW, dS);
        a.nextrap = first(c + 1) - first(c);
        a.denseF = dF + first(c) * depth;
        a.denseB = dB + first(c) * depth;
        a.image_shots = dI + (size_t)first(c) * nx;
        a.img_sstride = (long long)plane;
        IMG2D_CUDA(cudaMemsetAsync(plan.counter.p, 0, sizeof(int), 0));
        return launch_kernel(&plan, a, plan.grid, 0);
    });
    const cudaError_t done = cudaDeviceSynchronize();  // nothing queued is left behind, errors or not
    if (rc) return rc;
    IMG2D_CUDA(done);
    // rows [0, nextrap) of every shot image
    IMG2D_CUDA(cudaMemcpy2D(image, plane * sizeof(float), dI, plane * sizeof(float),
                            (size_t)nextrap * nx * sizeof(float), ns, cudaMemcpyDeviceToHost));
    if (write_back) {
        // only the first nf rows of every (nt, nx) shot block carry data
        IMG2D_CUDA(cudaMemcpy2D(wave, (size_t)nt * nx * sizeof(cpx), dW, (size_t)nt * nx * sizeof(cpx),
                                (size_t)nf * nx * sizeof(cpx), ns, cudaMemcpyDeviceToHost));
        IMG2D_CUDA(cudaMemcpy2D(shot, (size_t)nt * nx * sizeof(cpx), dS, (size_t)nt * nx * sizeof(cpx),
                                (size_t)nf * nx * sizeof(cpx), ns, cudaMemcpyDeviceToHost));
    }
    return IMG2D_OK;
}

// Per device: one cached plan for the host compact entry point, reused while the geometry is
// unchanged, and its device buffers, kept between calls (grown on demand) so a call allocates
// nothing when the sizes repeat.  Everything in an entry belongs to that device and is only used
// (and freed) while it is the current device.
struct HostEntryBuffers {
    DevBuf omega, vel, tabF, tabB, wave, shot, image, image_shots;
    // frequency-chunked path: items per chunk, the two queue counters and two status words, its
    // streams (copies in, copies out, two for the kernels); its two sets of per-CTA image partials
    // are the plan's partial buffers, grown to twice the single-launch size
    DevBuf chunk_items, pipe_counter;
    unsigned long long chunk_plan = 0;       // uid of the plan and chunk count chunk_items was built for
    int chunks = 0;
    std::vector<int> chunk_first;            // first item of each chunk, chunks + 1 entries
    cudaStream_t st[4] = {nullptr, nullptr, nullptr, nullptr};
    std::vector<cudaEvent_t> ev;
    ~HostEntryBuffers()
    {
        for (cudaEvent_t e : ev) cudaEventDestroy(e);
        for (cudaStream_t x : st)
            if (x) cudaStreamDestroy(x);
    }
};

// img2d_migrate_compact in C frequency chunks.  Each chunk's spectra go to the device, its items
// run as one persistent launch and its final wavefields come back, on separate streams, so the
// copies of one chunk overlap the kernels of the others.  The launches alternate between two
// streams, each with its own work-queue counter and its own set of per-CTA image partials: a
// launch's clusters start on the SMs that the previous launch's last items leave free, and the two
// partial sets are summed once at the end.  Each launch is issued before the wavefields of the
// previous chunk are copied back, so the GPU has queued work while a pageable copy holds the host.
// The kernels and the per-item arithmetic are those of a single launch.
static int migrate_chunked(img2d_plan *p, HostEntryBuffers &hb, int C, img2d_c64 *wave_fs, img2d_c64 *shot_fs,
                           cpx *dW, cpx *dS, float *dI)
{
    int rc;
    const int nf = p->nf;
    const size_t plane = (size_t)p->nextrap * p->nx;
    auto fbegin = [&](int c) { return (int)((long long)c * nf / C); };
    if (hb.chunk_plan != p->uid || hb.chunks != C) {
        // within a chunk, widest groups first (the short items end the launch)
        std::vector<int2> items;
        hb.chunk_first.assign(1, 0);
        for (int c = 0; c < C; ++c) {
            for (int g : p->group_order)
                for (int j = fbegin(c); j < fbegin(c + 1); ++j) items.push_back(make_int2(g, j));
            hb.chunk_first.push_back((int)items.size());
        }
        if ((rc = hb.chunk_items.ensure(items.size() * sizeof(int2)))) return rc;
        IMG2D_CUDA(cudaMemcpy(hb.chunk_items.p, items.data(), items.size() * sizeof(int2), cudaMemcpyHostToDevice));
        hb.chunk_plan = p->uid;
        hb.chunks = C;
    }
    const size_t set_bytes = (size_t)p->grid * plane * sizeof(float);
    if ((rc = p->partial.ensure(2 * set_bytes))) return rc;
    if ((rc = p->comp.ensure(2 * set_bytes))) return rc;
    if ((rc = hb.pipe_counter.ensure(4 * sizeof(int)))) return rc;
    if (p->rows && (rc = p->visits.ensure(2 * (size_t)p->grid * sizeof(int)))) return rc;
    for (cudaStream_t &x : hb.st)
        if (!x) IMG2D_CUDA(cudaStreamCreateWithFlags(&x, cudaStreamNonBlocking));
    while ((int)hb.ev.size() < 2 * C + 1) {
        cudaEvent_t e;
        IMG2D_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        hb.ev.push_back(e);
    }
    cudaStream_t sin = hb.st[0], sout = hb.st[1], sk[2] = {hb.st[2], hb.st[3]};
    int *cnt = hb.pipe_counter.as<int>();
    float *part = p->partial.as<float>(), *comp = p->comp.as<float>();
    // zeroed partial sets, counters and status words before the first launch of either stream
    if (p->rows) {
        IMG2D_CUDA(cudaMemsetAsync(p->visits.p, 0, 2 * (size_t)p->grid * sizeof(int), sk[0]));
    } else {
        IMG2D_CUDA(cudaMemsetAsync(part, 0, 2 * set_bytes, sk[0]));
        IMG2D_CUDA(cudaMemsetAsync(comp, 0, 2 * set_bytes, sk[0]));
    }
    IMG2D_CUDA(cudaMemsetAsync(cnt, 0, 4 * sizeof(int), sk[0]));
    IMG2D_CUDA(cudaEventRecord(hb.ev[2 * C], sk[0]));
    IMG2D_CUDA(cudaStreamWaitEvent(sk[1], hb.ev[2 * C], 0));
    auto copy_rows = [&](int c, bool in) -> int {
        const int f0 = fbegin(c), f1 = fbegin(c + 1);
        for (int s = 0; s < p->ns; ++s) {
            const long long off = p->off[s] + (long long)f0 * p->w[s];
            const size_t bytes = (size_t)(f1 - f0) * p->w[s] * sizeof(cpx);
            if (in) {
                IMG2D_CUDA(cudaMemcpyAsync(dW + off, wave_fs + off, bytes, cudaMemcpyHostToDevice, sin));
                IMG2D_CUDA(cudaMemcpyAsync(dS + off, shot_fs + off, bytes, cudaMemcpyHostToDevice, sin));
            } else {
                IMG2D_CUDA(cudaMemcpyAsync(wave_fs + off, dW + off, bytes, cudaMemcpyDeviceToHost, sout));
                IMG2D_CUDA(cudaMemcpyAsync(shot_fs + off, dS + off, bytes, cudaMemcpyDeviceToHost, sout));
            }
        }
        return IMG2D_OK;
    };
    const int K = std::max(1, p->cluster);
    for (int c = 0; c < C; ++c) {
        if ((rc = copy_rows(c, true))) return rc;
        IMG2D_CUDA(cudaEventRecord(hb.ev[2 * c], sin));
        cudaStream_t st = sk[c & 1];
        IMG2D_CUDA(cudaStreamWaitEvent(st, hb.ev[2 * c], 0));
        if (c >= 2) IMG2D_CUDA(cudaMemsetAsync(cnt + (c & 1), 0, sizeof(int), st));  // after launch c - 2
        MigrateArgs a = base_args(p, dW, dS);
        const int n = hb.chunk_first[c + 1] - hb.chunk_first[c];
        a.items = hb.chunk_items.as<int2>() + hb.chunk_first[c];
        a.n_items = n;
        a.counter = cnt + (c & 1);
        a.status = cnt + 2 + (c & 1);
        a.partial = dI ? part + (size_t)(c & 1) * p->grid * plane : nullptr;
        a.comp = dI ? comp + (size_t)(c & 1) * p->grid * plane : nullptr;
        a.visits = dI && p->rows ? p->visits.as<int>() + (size_t)(c & 1) * p->grid : nullptr;
        if ((rc = launch_kernel(p, a, std::min(n, p->grid / K) * K, st))) return rc;
        IMG2D_CUDA(cudaEventRecord(hb.ev[2 * c + 1], st));
        if (c >= 1) {
            IMG2D_CUDA(cudaStreamWaitEvent(sout, hb.ev[2 * c - 1], 0));
            if ((rc = copy_rows(c - 1, false))) return rc;
        }
    }
    IMG2D_CUDA(cudaStreamWaitEvent(sout, hb.ev[2 * C - 1], 0));
    if ((rc = copy_rows(C - 1, false))) return rc;
    if (dI) {
        IMG2D_CUDA(cudaStreamWaitEvent(sk[0], hb.ev[2 * C - 1], 0));
        if (C >= 2) IMG2D_CUDA(cudaStreamWaitEvent(sk[0], hb.ev[2 * C - 3], 0));
        const int blocks = (int)std::min<size_t>((plane + 31) / 32, 148 * 64);
        reduce_partials_kernel<<<blocks, 256, 0, sk[0]>>>(part, comp, p->rows ? p->visits.as<int>() : nullptr, 2 * p->grid,
                                                          (long long)plane, dI);
        IMG2D_CUDA(cudaGetLastError());
    }
    for (cudaStream_t x : hb.st) IMG2D_CUDA(cudaStreamSynchronize(x));
    int status[2] = {0, 0};
    IMG2D_CUDA(cudaMemcpy(status, cnt + 2, sizeof(status), cudaMemcpyDeviceToHost));
    if (status[0] || status[1])
        return fail(IMG2D_ECUDA, "a bounded wait in the migration kernel gave up: the results of that call are not valid");
    return IMG2D_OK;
}
struct HostCache {
    img2d_plan *plan = nullptr;
    std::vector<int> key;
    HostEntryBuffers *bufs = nullptr;
};
static std::mutex g_cache_mu;
static std::map<int, HostCache> g_host_cache;

}  // namespace img2d

// ---------------------------------------------------------------------------------------
// Fixed scratch for img2d_migrate_compact_noalloc.  A file-scope device array: every GPU that
// loads this library holds it (IMG2D_NOALLOC_SCRATCH_BYTES) until the process exits.  In host code
// the name g_noalloc_scratch is only a stand-in for the symbol, not a device address, so the
// address is looked up once per device with cudaGetSymbolAddress while that device is current.
// ---------------------------------------------------------------------------------------
static __device__ __align__(256) unsigned char g_noalloc_scratch[IMG2D_NOALLOC_SCRATCH_BYTES];

namespace img2d {

static std::mutex g_noalloc_mu;
static void *g_noalloc_addr[256];

static int noalloc_scratch(void **out)
{
    int dev = 0;
    IMG2D_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 256) return fail(IMG2D_EINVAL, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
        void *addr = nullptr;
        IMG2D_CUDA(cudaGetSymbolAddress(&addr, g_noalloc_scratch));
        g_noalloc_addr[dev] = addr;
    }
    *out = g_noalloc_addr[dev];
    return IMG2D_OK;
}

}  // namespace img2d

using namespace img2d;

extern "C" {

const char *img2d_last_error(void) { return g_err.c_str(); }

void img2d_set_alloc_limit(size_t max_bytes)
{
    std::lock_guard<std::mutex> lock(g_alloc_mu);
    g_alloc_limit = max_bytes;
    g_alloc_limit_set = true;
}

int img2d_version(void) { return 10000; }

int img2d_extrapolate_host_order(int ns, int nextrap, int nz, int nx, int nf, int nt, int M,
                                 const img2d_c64 *op_forw, const img2d_c64 *op_back,
                                 img2d_c64 *wave_fs, img2d_c64 *shot_fs, float *image)
{
    return run_dense(ns, nextrap, nz, nx, nf, nt, M, (const cpx *)op_forw, (const cpx *)op_back,
                     (cpx *)wave_fs, (cpx *)shot_fs, image, 1);
}

int img2d_extrapolate_device_order(int ns, int nextrap, int nz, int nt, int nf, int nx, int M,
                                   const img2d_c64 *op_forw, img2d_c64 *forw_pulse,
                                   const img2d_c64 *op_back, img2d_c64 *back_pulse, float *image,
                                   int write_back)
{
    return run_dense(ns, nextrap, nz, nx, nf, nt, M, (const cpx *)op_forw, (const cpx *)op_back,
                     (cpx *)forw_pulse, (cpx *)back_pulse, image, write_back);
}

int img2d_plan_create(img2d_plan **plan, int ns, int nextrap, int nz, int nx, int nf, int nt, int M,
                      int nk, const int *shot_x0, const int *shot_nx, int flags)
{
    if (!plan) return fail(IMG2D_EINVAL, "plan pointer is NULL");
    *plan = nullptr;
    int rc;
    if ((rc = check_device())) return rc;
    img2d_plan *p = new img2d_plan();
    const int mode = (flags & IMG2D_FLAG_TWO_TABLES) ? OP_TWO : OP_CONJ;
    if ((rc = build_plan(p, ns, nextrap, nz, nx, nf, nt, M, nk, shot_x0, shot_nx, flags, mode))) {
        delete p;
        return rc;
    }
    *plan = p;
    return IMG2D_OK;
}

int img2d_plan_set_model(img2d_plan *p, const double *d_omega, const double *d_velocity, double dk,
                         const img2d_c64 *d_tab_forw, const img2d_c64 *d_tab_back, void *stream)
{
    if (!p) return fail(IMG2D_EINVAL, "plan is NULL");
    return set_model(p, d_omega, d_velocity, dk, (const cpx *)d_tab_forw, (const cpx *)d_tab_back,
                     (cudaStream_t)stream);
}

int img2d_plan_execute(img2d_plan *p, img2d_c64 *d_wave, img2d_c64 *d_shot, float *d_image,
                       float *d_image_shots, void *stream)
{
    if (!p) return fail(IMG2D_EINVAL, "plan is NULL");
    if (!d_wave || !d_shot) return fail(IMG2D_EINVAL, "wavefield pointers are NULL");
    MigrateArgs a = base_args(p, (cpx *)d_wave, (cpx *)d_shot);
    return launch(p, a, d_image, d_image_shots, (long long)p->nz * p->nx, (cudaStream_t)stream);
}

int img2d_plan_demigrate(img2d_plan *p, const float *d_refl, const img2d_c64 *d_wave, img2d_c64 *d_data,
                         int slab_depth, int source_mode, void *stream)
{
    if (!p) return fail(IMG2D_EINVAL, "plan is NULL");
    if (!d_refl || !d_wave || !d_data) return fail(IMG2D_EINVAL, "null device pointer");
    if ((const void *)d_wave == (const void *)d_data) return fail(IMG2D_EINVAL, "data must not alias wave");
    if (p->mode != OP_CONJ) return fail(IMG2D_EINVAL, "demigration supports the single-table mode only");
    if (source_mode < IMG2D_SOURCE_RECOMPUTE || source_mode > IMG2D_SOURCE_REUSE)
        return fail(IMG2D_EINVAL, "source_mode must be IMG2D_SOURCE_RECOMPUTE, _KEEP or _REUSE");
    int rc;
    if ((rc = demig_prepare(p, slab_depth))) return rc;
    if (source_mode == IMG2D_SOURCE_REUSE && !p->adj_cache_valid)
        return fail(IMG2D_EINVAL, "no kept source checkpoints on this plan (call with IMG2D_SOURCE_KEEP first, "
                                  "after the last set_model, with the same slab depth)");
    int rows_grid = p->adj_grid;
    if (p->adj_rows) {
        rc = IMG2D_OK;
        if (source_mode == IMG2D_SOURCE_KEEP)
            rc = p->adj_cache.ensure(p->adj_full_cache ? (size_t)p->adj_items_n * p->adj_cache_item * sizeof(float2) : 16);
        if (!rc && !(p->adj_full_cache && source_mode != IMG2D_SOURCE_RECOMPUTE)) {
            rc = p->adj_work.ensure((size_t)rows_grid * p->adj_work_cta * sizeof(float2));
            // beside a kept source, which the slab kernel could not use: fewer CTAs
            while (rc == IMG2D_ENOMEM && p->adj_cache_valid && p->adj_full_cache && rows_grid > 1) {
                rows_grid /= 2;
                rc = p->adj_work.ensure((size_t)rows_grid * p->adj_work_cta * sizeof(float2));
            }
        }
        if (!rc) rc = p->tab_rows.ensure(rows_table_bytes(p));
        if (rc == IMG2D_ENOMEM && source_mode != IMG2D_SOURCE_REUSE) {
            // too little memory for every S_l: the slab kernel
            p->adj_cache.release();
            p->adj_work.release();
            p->adj_allow_rows = p->adj_rows = false;
            p->adj_rows_fn = nullptr;
            p->adj_slab = 0;
            rc = demig_prepare(p, slab_depth);
        }
        if (rc) return rc;
    }
    const long long cache_elems = (long long)p->adj_items_n * p->adj_cache_item;  // float2
    if (source_mode == IMG2D_SOURCE_KEEP && !p->adj_rows) {
        if ((rc = p->adj_cache.ensure((size_t)cache_elems * sizeof(float2)))) return rc;
    }
    cudaStream_t st = (cudaStream_t)stream;
    DemigrateArgs a{};
    a.nextrap = p->nextrap;
    a.nx = p->nx;
    a.M = p->M;
    a.tab_stride = p->tab_stride;
    a.n_items = p->adj_items_n;
    a.slab = p->adj_slab;
    a.nslab = p->adj_nslab;
    a.items = p->adj_items.as<int2>();
    a.groups = p->adj_groups.as<GroupDesc>();
    a.segs = p->adj_segs.as<int4>();
    a.owner = p->adj_owner.as<int16_t>();
    a.shot_off = p->shot_off.as<long long>();
    a.tab = p->tabF.as<cpx>();
    a.idx = p->idx.as<uint16_t>();
    a.idx_jstride = (long long)p->nextrap * p->idx_lstride;
    a.idx_lstride = p->idx_lstride;
    a.wave = (const cpx *)d_wave;
    a.refl = d_refl;
    a.data = (cpx *)d_data;
    a.work = p->adj_work.as<float2>();
    a.work_cta = p->adj_work_cta;
    a.wmax = p->adj_wmax;
    a.plane = p->adj_wide_fn ? demigw_share(p->adj_wmax, p->adj_cluster) : 0;
    a.counter = p->adj_counter.as<int>();
    a.ckpt_mode = source_mode;
    a.ckpt_items = source_mode == IMG2D_SOURCE_RECOMPUTE ? nullptr : p->adj_cache.as<float2>();
    IMG2D_CUDA(cudaMemsetAsync(p->adj_counter.p, 0, sizeof(int), st));
    p->launched = true;
    if (p->timing && !p->ev0) {
        IMG2D_CUDA(cudaEventCreate(&p->ev0));
        IMG2D_CUDA(cudaEventCreate(&p->ev1));
    }
    if (p->timing) IMG2D_CUDA(cudaEventRecord(p->ev0, st));
    if (p->adj_cluster) {
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = p->adj_cluster;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.gridDim = dim3(p->adj_grid, 1, 1);
        cfg.blockDim = dim3(p->adj_block, 1, 1);
        cfg.dynamicSmemBytes = p->adj_smem;
        cfg.stream = st;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        if (p->adj_wide_fn) {
            // its bounded waits report to the plan's status word
            IMG2D_CUDA(cudaLaunchKernelEx(&cfg, p->adj_wide_fn, a, p->counter.as<int>() + 1));
        } else {
            IMG2D_CUDA(cudaLaunchKernelEx(&cfg, p->adj_fn, a));
        }
    } else if (p->adj_rows) {
        if (!p->rows_tab_set && (rc = set_rows_table(p, st))) return rc;
        RowsAdjArgs ra{};
        ra.d = a;
        if (!p->adj_full_cache) ra.d.ckpt_mode = IMG2D_SOURCE_RECOMPUTE;
        ra.tab_rows = p->tab_rows.p;
        const RowsStarts &rs = plan_row_starts(p);
        for (int i = 0; i < 4; ++i) ra.row_start[i] = rs.s[i];
        ra.row_apart = rs.apart;
        ra.planes = ra.d.ckpt_mode ? p->adj_cache.p : p->adj_work.p;
        ra.plane = rows_adj_wp(p->adj_wmax);
        p->adj_rows_fn<<<rows_grid, p->adj_block, p->adj_smem, st>>>(ra);
    } else {
        p->adj_fn<<<p->adj_grid, p->adj_block, p->adj_smem, st>>>(a);
    }
    IMG2D_CUDA(cudaGetLastError());
    if (p->timing) {
        IMG2D_CUDA(cudaEventRecord(p->ev1, st));
        p->ev_recorded = true;
    }
    if (source_mode == IMG2D_SOURCE_KEEP) p->adj_cache_valid = true;
    return IMG2D_OK;
}

int img2d_plan_describe_demigration(const img2d_plan *p, char *buf, int buflen)
{
    if (!p || !buf || buflen <= 0) return fail(IMG2D_EINVAL, "bad describe arguments");
    if (!p->adj_fn && !p->adj_rows_fn && !p->adj_wide_fn) return fail(IMG2D_EINVAL, "no demigration has run on this plan yet");
    snprintf(buf, buflen,
             "{\"kernel\": \"%s\", \"cluster\": %d, \"G\": %d, \"X\": 8, \"L\": %d, \"grid\": %d, \"block\": %d, "
             "\"smem\": %zu, \"items\": %d, \"max_union_width\": %d, \"slab\": %d, \"slabs\": %d, "
             "\"workspace_bytes\": %zu, \"source_cache_bytes\": %zu, \"ring\": %s, \"wide\": %s}",
             p->adj_rows ? "demigrate_rows" : (p->adj_cluster ? "demigrate_cluster" : "demigrate"), p->adj_cluster, p->adj_G, p->L, p->adj_grid,
             p->adj_block, p->adj_smem, p->adj_items_n, p->adj_wmax, p->adj_slab,
             p->adj_nslab, p->adj_work.bytes, p->adj_cache.bytes, p->adj_ring ? "true" : "false", p->adj_wide_fn ? "true" : "false");
    return IMG2D_OK;
}

int img2d_plan_dense_table(const img2d_plan *p, int which, img2d_c64 *d_dense, void *stream)
{
    if (!p) return fail(IMG2D_EINVAL, "plan is NULL");
    if (!d_dense) return fail(IMG2D_EINVAL, "d_dense is NULL");
    if (which != 0 && which != 1) return fail(IMG2D_EINVAL, "which must be 0 (forward) or 1 (receiver)");
    if (p->mode == OP_DENSE) return fail(IMG2D_EINVAL, "a dense-table plan has no compact table");
    if (!p->model_set) return fail(IMG2D_EINVAL, "call img2d_plan_set_model first");
    if ((long long)p->nx * p->L >= (1ll << 31) || (long long)p->nextrap * p->nf >= (1ll << 31))
        return fail(IMG2D_EINVAL, "dense table rows too large");
    const bool back_rows = which == 1 && p->mode == OP_TWO;
    const cpx *tab = back_rows ? p->tabB.as<cpx>() : p->tabF.as<cpx>();
    const int conj = which == 1 && !back_rows;
    cudaStream_t st = (cudaStream_t)stream;
    dense_table_kernel<<<p->nextrap * p->nf, 256, 0, st>>>(p->idx.as<uint16_t>(), p->nf, p->nextrap, p->nx,
                                                          p->idx_lstride, tab, p->tab_stride, p->L, conj,
                                                          (cpx *)d_dense);
    IMG2D_CUDA(cudaGetLastError());
    return IMG2D_OK;
}

long long img2d_plan_shot_offset(const img2d_plan *p, int s)
{
    if (!p || s < 0 || s >= p->ns) return -1;
    return p->off[s];
}

long long img2d_plan_wavefield_elems(const img2d_plan *p) { return p ? p->wave_elems : -1; }

size_t img2d_plan_workspace_bytes(const img2d_plan *p)
{
    if (!p) return 0;
    return p->items.bytes + p->groups.bytes + p->segs.bytes + p->owner.bytes + p->shot_off.bytes +
           p->idx.bytes + p->tabF.bytes + p->tabB.bytes + p->tab16buf.bytes + p->tab_rows.bytes + p->partial.bytes +
           p->comp.bytes + p->visits.bytes + p->counter.bytes +
           p->naive_buf.bytes + p->adj_items.bytes + p->adj_groups.bytes + p->adj_segs.bytes + p->adj_owner.bytes +
           p->adj_work.bytes + p->adj_counter.bytes + p->adj_cache.bytes;
}

int img2d_plan_describe(const img2d_plan *p, char *buf, int buflen)
{
    if (!p || !buf || buflen <= 0) return fail(IMG2D_EINVAL, "bad describe arguments");
    snprintf(buf, buflen,
             "{\"kernel\": \"%s\", \"cluster\": %d, \"G\": %d, \"X\": %d, \"L\": %d, \"grid\": %d, \"block\": %d, "
             "\"smem\": %zu, \"items\": %d, \"slots\": %d, \"max_union_width\": %d, \"mode\": %d, \"variant\": %d, "
             "\"table\": \"%s\", \"packing\": \"%s\", \"cost_units\": %.3f, \"computed_per_useful\": %.4f}",
             p->kname, p->cluster, p->G, p->fixed ? kX : 4, p->L, p->grid, p->block, p->smem,
             p->n_items, p->n_slots, p->max_w, p->mode, p->variant,
             p->tab16 == 2 ? "bf16" : (p->tab16 == 1 ? "fp16" : "fp32"), p->packing, p->pack_cost,
             p->computed_per_useful);
    return IMG2D_OK;
}

void img2d_plan_destroy(img2d_plan *p) { delete p; }

int img2d_plan_kernel_ms(img2d_plan *p, float *ms)
{
    if (!p || !ms) return fail(IMG2D_EINVAL, "bad arguments");
    if (!p->ev_recorded) return fail(IMG2D_EINVAL, "no kernel launched on this plan yet");
    IMG2D_CUDA(cudaEventSynchronize(p->ev1));
    IMG2D_CUDA(cudaEventElapsedTime(ms, p->ev0, p->ev1));
    return IMG2D_OK;
}

int img2d_pack_shots(int ns, int nx, int M, const int *shot_x0, const int *shot_nx, int windows, int K,
                     int *group_of_shot, int *slot_of_shot, int *group_u0, int *group_w, int *n_groups,
                     double *cost_units)
{
    if (ns <= 0 || nx <= 0 || M < 0 || !shot_x0 || !shot_nx || !group_of_shot || !slot_of_shot || !n_groups)
        return fail(IMG2D_EINVAL, "img2d_pack_shots: invalid arguments");
    if (ns > 32767) return fail(IMG2D_EINVAL, "at most 32767 shots");
    img2d_plan pl;
    pl.ns = ns;
    pl.nx = nx;
    pl.M = M;
    pl.x0.assign(shot_x0, shot_x0 + ns);
    pl.w.assign(shot_nx, shot_nx + ns);
    int wmax = 0;
    for (int s = 0; s < ns; ++s) {
        if (pl.x0[s] < 0 || pl.w[s] <= 0 || pl.x0[s] + pl.w[s] > nx)
            return fail(IMG2D_EINVAL, "shot " + std::to_string(s) + " aperture outside [0, nx)");
        wmax = std::max(wmax, pl.w[s]);
    }
    const int Kmin = (wmax + WideShape::PC - 1) / WideShape::PC;
    std::vector<GroupDesc> groups;
    std::vector<int4> segs;
    std::vector<int16_t> owner;
    double cost = 0.0;
    if (windows) {
        if (K < Kmin) return fail(IMG2D_EINVAL, "K too small for the widest shot");
        cost = pack_windows_best(&pl, WideShape::G, K, groups, segs, owner);
        if (cost < 0.0) return fail(IMG2D_EINVAL, "a shot fits no window");
    } else {
        colour_slots(&pl);
        const int widest = pack_groups(&pl, WideShape::G, groups, segs, owner);
        if (K <= 0) K = (widest + WideShape::PC - 1) / WideShape::PC;
        if (K * WideShape::PC < widest) return fail(IMG2D_EINVAL, "K too small for the widest group");
        for (const GroupDesc &g : groups) cost += wide_item_cost(g.W, K);
    }
    for (size_t g = 0; g < groups.size(); ++g) {
        if (group_u0) group_u0[g] = groups[g].u0;
        if (group_w) group_w[g] = groups[g].W;
        for (int k = groups[g].seg_begin; k < groups[g].seg_begin + groups[g].nseg; ++k) {
            group_of_shot[segs[k].x] = (int)g;
            slot_of_shot[segs[k].x] = segs[k].y;
        }
    }
    *n_groups = (int)groups.size();
    if (cost_units) *cost_units = cost;
    return IMG2D_OK;
}

int img2d_plan_status(img2d_plan *p, void *stream)
{
    if (!p) return fail(IMG2D_EINVAL, "plan is NULL");
    if (!p->launched) return fail(IMG2D_EINVAL, "no kernel launched on this plan yet");
    return img2d::read_status(p, (cudaStream_t)stream);
}

int img2d_plan_inject_status(img2d_plan *p, int status, void *stream)
{
    if (!p) return fail(IMG2D_EINVAL, "plan is NULL");
    IMG2D_CUDA(cudaMemcpyAsync(p->counter.as<int>() + 1, &status, sizeof(int), cudaMemcpyHostToDevice, (cudaStream_t)stream));
    IMG2D_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    return IMG2D_OK;
}

int img2d_measure_fp32_peak(double *tflops)
{
    if (!tflops) return fail(IMG2D_EINVAL, "tflops is NULL");
    int rc;
    if ((rc = check_device())) return rc;
    int dev = 0, nsm = 0;
    IMG2D_CUDA(cudaGetDevice(&dev));
    IMG2D_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    Scratch sc;
    float *out;
    const int blocks = nsm * 4, threads = 512, iters = 4096;
    if ((rc = sc.alloc(&out, (size_t)blocks * threads * sizeof(float)))) return rc;
    fma_probe_kernel<<<blocks, threads>>>(out, 64);
    IMG2D_CUDA(cudaGetLastError());
    cudaEvent_t e0, e1;
    IMG2D_CUDA(cudaEventCreate(&e0));
    IMG2D_CUDA(cudaEventCreate(&e1));
    float best = 1e30f;
    for (int r = 0; r < 3; ++r) {
        cudaEventRecord(e0);
        fma_probe_kernel<<<blocks, threads>>>(out, iters);
        cudaEventRecord(e1);
        cudaError_t e = cudaEventSynchronize(e1);
        if (e != cudaSuccess) {
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
            return fail(IMG2D_ECUDA, std::string("fma probe: ") + cudaGetErrorString(e));
        }
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        best = std::min(best, ms);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    // 16 chains x 8 FMAs per iteration per thread, 2 flops per FMA
    *tflops = 2.0 * 128.0 * iters * (double)blocks * threads / (best * 1e-3) * 1e-12;
    return IMG2D_OK;
}

int img2d_ricker_sources(int ns, int nt, int nx, double dt, double x_first, double dx, double depth_offset,
                         double v, double fpeak, const double *src_x, float *d_out, void *stream)
{
    int rc;
    if ((rc = check_device())) return rc;
    if (ns <= 0 || nt <= 0 || nx <= 0 || !(dt > 0.0) || !(dx > 0.0) || !(v > 0.0))
        return fail(IMG2D_EINVAL, "invalid source-wavelet dimensions or spacing");
    if (!src_x || !d_out) return fail(IMG2D_EINVAL, "null pointer argument");
    cudaStream_t st = (cudaStream_t)stream;
    Scratch sc;
    double *d_sx;
    if ((rc = sc.alloc(&d_sx, (size_t)ns * sizeof(double)))) return rc;
    IMG2D_CUDA(cudaMemcpyAsync(d_sx, src_x, (size_t)ns * sizeof(double), cudaMemcpyHostToDevice, st));
    const long long total = (long long)ns * nt * nx;
    const int blocks = (int)std::min<long long>((total + 255) / 256, 148 * 32);
    ricker_sources_kernel<<<blocks, 256, 0, st>>>(ns, nt, nx, dt, x_first, dx, depth_offset, v, fpeak, d_sx, d_out);
    IMG2D_CUDA(cudaGetLastError());
    IMG2D_CUDA(cudaStreamSynchronize(st));  // the source positions are freed on return
    return IMG2D_OK;
}

// Apertures of a front-end call: per-shot start, width and offset of the packed block.
static int spectra_layout(int ns, int nt, int nx, int nf, int nt_rows, const int *shot_x0, const int *shot_nx,
                          std::vector<int> &x0, std::vector<int> &w, std::vector<long long> &off)
{
    if (ns <= 0 || nt <= 0 || nx <= 0 || nf <= 0 || nf > nt || nt_rows < nf)
        return fail(IMG2D_EINVAL, "invalid dimensions (need ns, nt, nx > 0, 0 < nf <= nt, nt_rows >= nf)");
    x0.assign(ns, 0);
    w.assign(ns, nx);
    off.assign(ns, 0);
    long long acc = 0;
    for (int s = 0; s < ns; ++s) {
        if (shot_x0) x0[s] = shot_x0[s];
        if (shot_nx) w[s] = shot_nx[s];
        if (x0[s] < 0 || w[s] <= 0 || x0[s] + w[s] > nx)
            return fail(IMG2D_EINVAL, "shot " + std::to_string(s) + " aperture outside [0, nx)");
        off[s] = acc;
        acc += (long long)nt_rows * w[s];
    }
    return IMG2D_OK;
}

// Front-end scratch of one device (transform tables, cuFFT spectra), kept and grown on demand.  A
// call holds the lock until its work has finished, so that the scratch has one user.
struct FrontScratch {
    DevBuf tables, spec;
    std::map<std::vector<long long>, cufftHandle> plans;  // by (nt, nx)
};
static std::mutex g_front_mu;
static std::map<int, FrontScratch> g_front;

// The two-stage transform of records of nt samples: the divisor N1 <= 31 with the fewest
// multiply-adds per trace; none (N1 = 0) where that exceeds 150 nt (a prime nt: cuFFT is taken) or the
// inner sums of 8 traces do not fit in shared memory.  16 traces per CTA (64-byte reads) unless only 8
// leave room for two CTAs per SM.
static SpecPlan spec_plan(int nt, int nf, size_t smem_optin, double &best_cost)
{
    SpecPlan best{};
    best_cost = 150.0 * nt;
    for (int N1 = 1; N1 <= 31 && N1 <= nt; ++N1) {
        if (nt % N1) continue;
      for (int M : {8, 10}) {
        SpecPlan p{};
        p.M = M;
        p.N1 = N1;
        p.N2 = nt / N1;
        p.K1 = N1 / 2 + 1;
        p.mp = ((nf + N1 - 1) / N1 + M - 1) / M * M;
        const size_t per = (size_t)p.N2 * p.K1 * sizeof(float2), table = (size_t)p.N2 * p.mp * sizeof(float2);
        p.bs = table <= 8192;
        const size_t more = p.bs ? table : 0, room = smem_optin - 6144;
        p.C = 16 * per + more <= room / 2 ? 16 : (8 * per + more <= room / 2 ? 8 : (16 * per + more <= room ? 16 : 8));
        p.smem = per * p.C + more;
        if (p.smem > room) continue;
        double cost = 2.0 * ((p.K1 + kSpecKC - 1) / kSpecKC * kSpecKC) * p.N2 * (N1 / 2);
        for (int k1 = 0; k1 < std::min(N1, nf); ++k1) cost += 4.0 * p.N2 * ((nf - 1 - k1) / (N1 * M) + 1) * M;
        if (cost < best_cost) {
            best_cost = cost;
            best = p;
        }
      }
    }
    // a few tasks in the second stage: their sums in parts of whole blocks, as many as there are threads for
    // and as the inner sums' place holds partial sums
    best.S = 1;
    best.T2 = best.N2;
    if (best.N1) {
        const int tasks = std::min(best.N1, nf) * (best.mp / best.M);
        const int parts = std::min(256 / (best.C / 2) / tasks, best.N2 * best.K1 / (tasks * best.M));
        if (parts >= 4) {
            best.T2 = ((best.N2 + parts - 1) / parts + kSpecBlock - 1) / kSpecBlock * kSpecBlock;
            best.S = (best.N2 + best.T2 - 1) / best.T2;
        }
    }
    return best;
}

static SpecShots spec_shots(int s0, int n, const std::vector<int> &x0, const std::vector<int> &w,
                            const std::vector<long long> &off)
{
    SpecShots sh{};
    for (int i = 0; i < n; ++i) {
        sh.x0[i] = x0[s0 + i];
        sh.w[i] = w[s0 + i];
        sh.off[i] = off[s0 + i];
    }
    return sh;
}

// cuFFT path: the real-to-complex transforms along time of groups of shots, then the packing kernel.
static int spectra_by_cufft(FrontScratch &fs, int ns, int nt, int nx, int nf, const float *d_records,
                            const std::vector<int> &x0, const std::vector<int> &w, const std::vector<long long> &off,
                            cpx *d_out, cudaStream_t st)
{
    int rc;
    // shots per transform group: their spectra (nt/2+1 rows) in at most 512 MB of scratch
    const long long shot_spec = (long long)(nt / 2 + 1) * nx;
    const int group = (int)std::max<long long>(1, std::min<long long>(ns, (512ll << 20) / (shot_spec * 8)));
    // One plan per (nt, nx), kept for the process: the nx transforms of length nt of one shot,
    // element (t, x) at x + t*nx in and at x + j*nx out; shots are issued one by one.
    const std::vector<long long> key = {nt, nx};
    auto itp = fs.plans.find(key);
    if (itp == fs.plans.end()) {
        int n[1] = {nt};
        int inembed[1] = {nt}, onembed[1] = {nt / 2 + 1};
        cufftHandle h;
        if (cufftCreate(&h) != CUFFT_SUCCESS) return fail(IMG2D_ECUDA, "cufftCreate failed");
        size_t ws = 0;
        if (cufftMakePlanMany(h, 1, n, inembed, nx, 1, onembed, nx, 1, CUFFT_R2C, nx, &ws) != CUFFT_SUCCESS) {
            cufftDestroy(h);
            return fail(IMG2D_ECUDA, "cufftMakePlanMany (real-to-complex along time) failed");
        }
        itp = fs.plans.emplace(key, h).first;
    }
    const cufftHandle plan = itp->second;
    if (cufftSetStream(plan, st) != CUFFT_SUCCESS) return fail(IMG2D_ECUDA, "cufftSetStream failed");
    // cuFFT reads 8-byte pairs: a shot whose records start between two goes through an aligned copy (with
    // an odd nt * nx every other one; all of them or the others where the caller's array itself does)
    auto between = [&](int s) { return (reinterpret_cast<uintptr_t>(d_records + (long long)s * nt * nx) & 7) != 0; };
    const bool copies = between(0) || (ns > 1 && between(1));
    if ((rc = fs.spec.ensure((size_t)group * shot_spec * sizeof(cpx) + (copies ? (size_t)nt * nx * sizeof(float) : 0)))) return rc;
    cpx *d_spec = fs.spec.as<cpx>();
    float *aligned = reinterpret_cast<float *>(d_spec + (long long)group * shot_spec);
    Scratch sc;
    int *d_x0, *d_w;
    long long *d_off;
    if ((rc = sc.alloc(&d_x0, ns * sizeof(int)))) return rc;
    if ((rc = sc.alloc(&d_w, ns * sizeof(int)))) return rc;
    if ((rc = sc.alloc(&d_off, ns * sizeof(long long)))) return rc;
    IMG2D_CUDA(cudaMemcpyAsync(d_x0, x0.data(), ns * sizeof(int), cudaMemcpyHostToDevice, st));
    IMG2D_CUDA(cudaMemcpyAsync(d_w, w.data(), ns * sizeof(int), cudaMemcpyHostToDevice, st));
    IMG2D_CUDA(cudaMemcpyAsync(d_off, off.data(), ns * sizeof(long long), cudaMemcpyHostToDevice, st));
    for (int s0 = 0; s0 < ns; s0 += group) {
        const int nsc = std::min(group, ns - s0);
        for (int k = 0; k < nsc; ++k) {
            cufftReal *in = const_cast<cufftReal *>(d_records + (long long)(s0 + k) * nt * nx);
            if (between(s0 + k)) {
                IMG2D_CUDA(cudaMemcpyAsync(aligned, in, (size_t)nt * nx * sizeof(float), cudaMemcpyDeviceToDevice, st));
                in = aligned;
            }
            cufftComplex *o = reinterpret_cast<cufftComplex *>(d_spec + (long long)k * shot_spec);
            if (cufftExecR2C(plan, in, o) != CUFFT_SUCCESS) return fail(IMG2D_ECUDA, "cufftExecR2C failed");
        }
        const long long total = (long long)nsc * nf * nx;
        const int blocks = (int)std::min<long long>((total + 255) / 256, 148 * 32);
        pack_spectra_kernel<<<blocks, 256, 0, st>>>(s0, nsc, nt, nx, nf, d_spec, d_x0, d_w, d_off, d_out);
        IMG2D_CUDA(cudaGetLastError());
    }
    IMG2D_CUDA(cudaStreamSynchronize(st));  // the descriptors are freed on return
    return IMG2D_OK;
}

int img2d_records_to_spectra(int ns, int nt, int nx, int nf, int nt_rows, const float *d_records,
                             const int *shot_x0, const int *shot_nx, img2d_c64 *d_out, void *stream)
{
    int rc;
    if ((rc = check_device())) return rc;
    std::vector<int> x0, w;
    std::vector<long long> off;
    if ((rc = spectra_layout(ns, nt, nx, nf, nt_rows, shot_x0, shot_nx, x0, w, off))) return rc;
    if (!d_records || !d_out) return fail(IMG2D_EINVAL, "null pointer argument");
    cudaStream_t st = (cudaStream_t)stream;
    int dev = 0, smem_optin = 0;
    IMG2D_CUDA(cudaGetDevice(&dev));
    IMG2D_CUDA(cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    std::lock_guard<std::mutex> lock(g_front_mu);
    FrontScratch &fs = g_front[dev];
    double cost;
    const SpecPlan pl = spec_plan(nt, nf, (size_t)smem_optin, cost);
    // cuFFT transforms all nx traces to all rows: about 0.5 ms of launches and 8.5 ps per sample.  It
    // is the faster one where most rows of many full-width records are kept (256 x 1024 x 2048 samples
    // to 512 rows: 6.0 ms here, 5.0 ms with cuFFT; 32 x 1024 x 1024 to 512 rows: 0.43 and 1.0 ms).
    double traces = 0.0;
    for (int x : w) traces += x;
    const bool library = 8.2e-11 * cost * traces > 0.5 + 8.5e-9 * ns * nt * (double)nx;
    if (!pl.N1 || library) return spectra_by_cufft(fs, ns, nt, nx, nf, d_records, x0, w, off, (cpx *)d_out, st);
    const size_t n1 = (size_t)kSpecK * kSpecK, n2 = (size_t)pl.N2 * pl.mp, n3 = (size_t)nt;
    if ((rc = fs.tables.ensure((n1 + n2 + n3) * sizeof(float2)))) return rc;
    float2 *T1 = fs.tables.as<float2>(), *B = T1 + n1, *A = B + n2;
    spec_tables_kernel<<<(int)std::min<size_t>((n1 + n2 + n3 + 255) / 256, 148 * 4), 256, 0, st>>>(pl, nt, T1, B, A);
    IMG2D_CUDA(cudaGetLastError());
#define IMG2D_SPEC(C, M)                                                                                       \
    (pl.S > 1 ? (pl.bs ? record_spectra_kernel<C, M, true, true> : record_spectra_kernel<C, M, false, true>)   \
              : (pl.bs ? record_spectra_kernel<C, M, true, false> : record_spectra_kernel<C, M, false, false>))
    auto kernel = pl.C == 16 ? (pl.M == 8 ? IMG2D_SPEC(16, 8) : IMG2D_SPEC(16, 10))
                             : (pl.M == 8 ? IMG2D_SPEC(8, 8) : IMG2D_SPEC(8, 10));
#undef IMG2D_SPEC
    IMG2D_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pl.smem));
    for (int s0 = 0; s0 < ns; s0 += kSpecShots) {
        const int n = std::min(kSpecShots, ns - s0);
        kernel<<<dim3((nx + pl.C - 1) / pl.C, n), 256, pl.smem, st>>>(pl, spec_shots(s0, n, x0, w, off), s0, nt, nx, nf,
                                                                      d_records, T1, B, A, (cpx *)d_out);
        IMG2D_CUDA(cudaGetLastError());
    }
    IMG2D_CUDA(cudaStreamSynchronize(st));
    return IMG2D_OK;
}

int img2d_source_spectra(int ns, int nt, int nx, int nf, int nt_rows, double dt, double x_first, double dx,
                         double depth_offset, double v, double fpeak, const double *src_x, const int *shot_x0,
                         const int *shot_nx, img2d_c64 *d_out, void *stream)
{
    int rc;
    if ((rc = check_device())) return rc;
    if (!(dt > 0.0) || !(dx > 0.0) || !(v > 0.0))
        return fail(IMG2D_EINVAL, "invalid source-wavelet dimensions or spacing");
    std::vector<int> x0, w;
    std::vector<long long> off;
    if ((rc = spectra_layout(ns, nt, nx, nf, nt_rows, shot_x0, shot_nx, x0, w, off))) return rc;
    if (!src_x || !d_out) return fail(IMG2D_EINVAL, "null pointer argument");
    cudaStream_t st = (cudaStream_t)stream;
    // half width of the samples that are not zero in float32: (pi fpeak t)^2 = 150
    const double tw = std::sqrt(150.0) / (3.141592653589793 * std::fabs(fpeak));
    const double span = 2.0 * tw / dt + 3.0;
    if (span > 384.0 || !(span > 0.0)) {
        // a wavelet of more samples (or a constant): through the time domain
        float *d_t = nullptr;
        Scratch sc;
        if ((rc = sc.alloc(&d_t, (size_t)ns * nt * nx * sizeof(float)))) return rc;
        if ((rc = img2d_ricker_sources(ns, nt, nx, dt, x_first, dx, depth_offset, v, fpeak, src_x, d_t, stream))) return rc;
        return img2d_records_to_spectra(ns, nt, nx, nf, nt_rows, d_t, shot_x0, shot_nx, d_out, stream);
    }
    const int nsup = std::min(nt, (int)span), kp = (nf + kSrcK - 1) / kSrcK * kSrcK;
    int dev = 0, nsm = 0;
    IMG2D_CUDA(cudaGetDevice(&dev));
    IMG2D_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    std::lock_guard<std::mutex> lock(g_front_mu);
    FrontScratch &fs = g_front[dev];
    const size_t nw = ((size_t)nt + 1) / 2 * 2, nu = (size_t)nsup * kp;
    if ((rc = fs.tables.ensure((nw + nu) * sizeof(float2)))) return rc;
    float2 *W = fs.tables.as<float2>(), *U = W + nw;
    source_tables_kernel<<<(int)std::min<size_t>((nw + nu + 255) / 256, 148 * 4), 256, 0, st>>>(nt, (int)nw, nsup, kp, W, U);
    IMG2D_CUDA(cudaGetLastError());
    const size_t smem = (size_t)nsup * kSrcCols * sizeof(float);
    IMG2D_CUDA(cudaFuncSetAttribute(source_spectra_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    for (int s0 = 0; s0 < ns; s0 += kSpecShots) {
        const int n = std::min(kSpecShots, ns - s0);
        SpecShots sh = spec_shots(s0, n, x0, w, off);
        for (int i = 0; i < n; ++i) sh.sx[i] = src_x[s0 + i];
        // the 64 rows that a CTA takes at a time are shared out over two CTAs, over more where the
        // SMs would be left without (each forms the wavelets anew)
        const int cols = (nx + kSrcCols - 1) / kSrcCols;
        const int parts = std::min((nf + 63) / 64, std::max(2, 2 * nsm / (cols * n)));
        source_spectra_kernel<<<dim3(cols, n, parts), 256, smem, st>>>(sh, nt, nx, nf, nsup, kp, dt, x_first, dx,
                                                                         depth_offset, v, fpeak, tw, W, U, (cpx *)d_out);
        IMG2D_CUDA(cudaGetLastError());
    }
    IMG2D_CUDA(cudaStreamSynchronize(st));
    return IMG2D_OK;
}

int img2d_measure_l2_bandwidth(double *gbs)
{
    if (!gbs) return fail(IMG2D_EINVAL, "gbs is NULL");
    int rc;
    if ((rc = check_device())) return rc;
    int dev = 0, nsm = 0;
    IMG2D_CUDA(cudaGetDevice(&dev));
    IMG2D_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    Scratch sc;
    const long long bytes = 32ll << 20;  // resident in L2 (126 MB on B200)
    const long long n4 = bytes / 16;
    const int blocks = nsm * 4, threads = 512, iters = 64;
    float4 *buf;
    float *out;
    if ((rc = sc.alloc(&buf, (size_t)bytes))) return rc;
    if ((rc = sc.alloc(&out, (size_t)blocks * threads * sizeof(float)))) return rc;
    IMG2D_CUDA(cudaMemset(buf, 0, (size_t)bytes));
    l2_read_probe_kernel<<<blocks, threads>>>(buf, n4, 2, out);  // warm the lines into L2
    IMG2D_CUDA(cudaGetLastError());
    cudaEvent_t e0, e1;
    IMG2D_CUDA(cudaEventCreate(&e0));
    IMG2D_CUDA(cudaEventCreate(&e1));
    float best = 1e30f;
    for (int r = 0; r < 3; ++r) {
        cudaEventRecord(e0);
        l2_read_probe_kernel<<<blocks, threads>>>(buf, n4, iters, out);
        cudaEventRecord(e1);
        cudaError_t e = cudaEventSynchronize(e1);
        if (e != cudaSuccess) {
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
            return fail(IMG2D_ECUDA, std::string("l2 probe: ") + cudaGetErrorString(e));
        }
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        best = std::min(best, ms);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    *gbs = (double)bytes * iters / (best * 1e-3) * 1e-9;
    return IMG2D_OK;
}

int img2d_plan_execute_naive(img2d_plan *p, img2d_c64 *d_wave, img2d_c64 *d_shot, float *d_image,
                             void *stream)
{
    if (!p) return fail(IMG2D_EINVAL, "plan is NULL");
    if (p->mode != OP_CONJ) return fail(IMG2D_EINVAL, "naive form supports the single-table mode only");
    if (!d_wave || !d_shot || !d_image) return fail(IMG2D_EINVAL, "null device pointer");
    cudaStream_t st = (cudaStream_t)stream;
    const int M = p->M;
    const int maxw = *std::max_element(p->w.begin(), p->w.end());
    int rc;
    if ((rc = p->naive_buf.ensure(2 * (size_t)(maxw + 2 * M) * sizeof(float4)))) return rc;
    float4 *b0 = p->naive_buf.as<float4>(), *b1 = b0 + (maxw + 2 * M);
    IMG2D_CUDA(cudaMemsetAsync(d_image, 0, (size_t)p->nextrap * p->nx * sizeof(float), st));
    for (int s = 0; s < p->ns; ++s) {
        const int w = p->w[s], x0 = p->x0[s];
        const int blocks = (w + 127) / 128;
        for (int j = 0; j < p->nf; ++j) {
            IMG2D_CUDA(cudaMemsetAsync(b0, 0, 2 * (size_t)(maxw + 2 * M) * sizeof(float4), st));
            cpx *ws = (cpx *)d_wave + p->off[s] + (long long)j * w;
            cpx *rs = (cpx *)d_shot + p->off[s] + (long long)j * w;
            naive_pack_kernel<<<blocks, 128, 0, st>>>(ws, rs, w, M, b0, 1);
            float4 *cur = b0, *nxt = b1;
            for (int l = 0; l < p->nextrap; ++l) {
                const uint16_t *idx_row = p->idx.as<uint16_t>() + ((long long)j * p->nextrap + l) * p->idx_lstride;
                naive_step_kernel<<<blocks, 128, 0, st>>>(cur, nxt, w, M, p->tabF.as<cpx>(), p->tab_stride, idx_row,
                                                          x0, d_image + (long long)l * p->nx);
                std::swap(cur, nxt);
            }
            naive_unpack_kernel<<<blocks, 128, 0, st>>>(cur, w, M, ws, rs);
        }
    }
    IMG2D_CUDA(cudaGetLastError());
    return IMG2D_OK;
}

int img2d_migrate_compact_noalloc(int ns, int nextrap, int nz, int nx, int nf, int nt, int M, int nk, double dk,
                                  const double *d_omega, const double *d_velocity, const img2d_c64 *d_tab_forw,
                                  const int *shot_x0, const int *shot_nx, img2d_c64 *d_wave, img2d_c64 *d_shot,
                                  float *d_image, void *stream)
{
    int rc;
    if ((rc = check_device())) return rc;
    if (!d_omega || !d_velocity || !d_tab_forw || !d_wave || !d_shot || !d_image)
        return fail(IMG2D_EINVAL, "null pointer argument");
    void *base = nullptr;
    if ((rc = noalloc_scratch(&base))) return rc;
    Carver carver;
    carver.base = static_cast<unsigned char *>(base);
    carver.cap = IMG2D_NOALLOC_SCRATCH_BYTES;
    img2d_plan plan;
    plan.carver = &carver;
    plan.upload_stream = (cudaStream_t)stream;
    plan.timing = false;
    for (DevBuf *b : {&plan.items, &plan.groups, &plan.segs, &plan.owner, &plan.shot_off, &plan.idx, &plan.tabF,
                      &plan.tabB, &plan.tab16buf, &plan.partial, &plan.comp, &plan.counter, &plan.naive_buf})
        b->carver = &carver;
    if ((rc = build_plan(&plan, ns, nextrap, nz, nx, nf, nt, M, nk, shot_x0, shot_nx, IMG2D_FLAG_NO_CLUSTER, OP_CONJ)))
        return rc;
    cudaStream_t st = (cudaStream_t)stream;
    if ((rc = set_model(&plan, d_omega, d_velocity, dk, (const cpx *)d_tab_forw, nullptr, st))) return rc;
    MigrateArgs a = base_args(&plan, (cpx *)d_wave, (cpx *)d_shot);
    return launch(&plan, a, d_image, nullptr, 0, st);
}

void img2d_release_host_cache(void)
{
    std::lock_guard<std::mutex> lock(g_cache_mu);
    int cur = -1;
    if (cudaGetDevice(&cur) != cudaSuccess) {
        cudaGetLastError();
        cur = -1;
    }
    for (auto &kv : g_host_cache) {
        // free each device's plan and buffers with that device current
        if (cudaSetDevice(kv.first) != cudaSuccess) cudaGetLastError();
        delete kv.second.plan;
        delete kv.second.bufs;
    }
    g_host_cache.clear();
    std::vector<int> devs;
    {
        DevicePool &pool = device_pool();
        std::lock_guard<std::mutex> plock(pool.mu);
        for (const auto &kv : pool.blocks) devs.push_back(kv.first);
    }
    for (int d : devs) pool_flush(d);
    {
        StageRing &ring = stage_ring();
        std::lock_guard<std::mutex> rlock(ring.mu);
        if (ring.host) cudaFreeHost(ring.host);
        ring.host = nullptr;
    }
    if (cur >= 0 && cudaSetDevice(cur) != cudaSuccess) cudaGetLastError();
}

int img2d_host_cache_device_count(void)
{
    std::lock_guard<std::mutex> lock(g_cache_mu);
    return (int)g_host_cache.size();
}

int img2d_migrate_compact(int ns, int nextrap, int nz, int nx, int nf, int nt, int M, int nk, double dk,
                          const double *omega, const double *velocity, const img2d_c64 *tab_forw,
                          const img2d_c64 *tab_back, const int *shot_x0, const int *shot_nx,
                          img2d_c64 *wave_fs, img2d_c64 *shot_fs, float *image, float *image_shots, int flags)
{
    int rc;
    if ((rc = check_device())) return rc;
    if (!omega || !velocity || !tab_forw || !wave_fs || !shot_fs)
        return fail(IMG2D_EINVAL, "null pointer argument");
    if ((flags & IMG2D_FLAG_TWO_TABLES) && !tab_back) return fail(IMG2D_EINVAL, "two-table mode needs tab_back");
    std::lock_guard<std::mutex> lock(g_cache_mu);
    int dev = 0;
    IMG2D_CUDA(cudaGetDevice(&dev));
    HostCache &hc = g_host_cache[dev];
    std::vector<int> key = {ns, nextrap, nz, nx, nf, nt, M, nk, flags};
    for (int s = 0; s < ns; ++s) {
        key.push_back(shot_x0 ? shot_x0[s] : 0);
        key.push_back(shot_nx ? shot_nx[s] : nx);
    }
    if (!hc.plan || key != hc.key) {
        delete hc.plan;
        hc.plan = nullptr;
        hc.key.clear();
        img2d_plan *p = nullptr;
        if ((rc = img2d_plan_create(&p, ns, nextrap, nz, nx, nf, nt, M, nk, shot_x0, shot_nx, flags))) return rc;
        hc.plan = p;
        hc.key = key;
    }
    img2d_plan *p = hc.plan;
    if (!hc.bufs) hc.bufs = new HostEntryBuffers();
    HostEntryBuffers &hb = *hc.bufs;
    const size_t L = 2 * (size_t)M + 1;
    const size_t plane = (size_t)nz * nx;
    if ((rc = hb.omega.ensure(nf * sizeof(double)))) return rc;
    if ((rc = hb.vel.ensure((size_t)nextrap * nx * sizeof(double)))) return rc;
    if ((rc = hb.tabF.ensure(nk * L * sizeof(cpx)))) return rc;
    if ((flags & IMG2D_FLAG_TWO_TABLES) && (rc = hb.tabB.ensure(nk * L * sizeof(cpx)))) return rc;
    if ((rc = hb.wave.ensure(p->wave_elems * sizeof(cpx)))) return rc;
    if ((rc = hb.shot.ensure(p->wave_elems * sizeof(cpx)))) return rc;
    if (image && (rc = hb.image.ensure((size_t)nextrap * nx * sizeof(float)))) return rc;
    if (image_shots && (rc = hb.image_shots.ensure((size_t)ns * plane * sizeof(float)))) return rc;
    double *dO = hb.omega.as<double>(), *dV = hb.vel.as<double>();
    cpx *dTF = hb.tabF.as<cpx>(), *dTB = (flags & IMG2D_FLAG_TWO_TABLES) ? hb.tabB.as<cpx>() : nullptr;
    cpx *dW = hb.wave.as<cpx>(), *dS = hb.shot.as<cpx>();
    float *dI = image ? hb.image.as<float>() : nullptr, *dIS = image_shots ? hb.image_shots.as<float>() : nullptr;
    IMG2D_CUDA(cudaMemcpy(dO, omega, nf * sizeof(double), cudaMemcpyHostToDevice));
    IMG2D_CUDA(cudaMemcpy(dV, velocity, (size_t)nextrap * nx * sizeof(double), cudaMemcpyHostToDevice));
    IMG2D_CUDA(cudaMemcpy(dTF, tab_forw, nk * L * sizeof(cpx), cudaMemcpyHostToDevice));
    if (dTB) IMG2D_CUDA(cudaMemcpy(dTB, tab_back, nk * L * sizeof(cpx), cudaMemcpyHostToDevice));
    // large wavefields: frequency chunks whose copies overlap the other chunks' kernels
    const int chunks = std::min(8, nf);
    if (!image_shots && chunks >= 2 && p->wave_elems * sizeof(cpx) >= ((size_t)64 << 20)) {
        if ((rc = set_model(p, dO, dV, dk, dTF, dTB, 0))) return rc;
        IMG2D_CUDA(cudaDeviceSynchronize());
        if ((rc = migrate_chunked(p, hb, chunks, wave_fs, shot_fs, dW, dS, dI))) {
            // leave no queued work behind on the error path
            for (cudaStream_t x : hb.st)
                if (x && cudaStreamSynchronize(x) != cudaSuccess) cudaGetLastError();
            return rc;
        }
        if (image) IMG2D_CUDA(cudaMemcpy(image, dI, (size_t)nextrap * nx * sizeof(float), cudaMemcpyDeviceToHost));
        return IMG2D_OK;
    }
    IMG2D_CUDA(cudaMemcpy(dW, wave_fs, p->wave_elems * sizeof(cpx), cudaMemcpyHostToDevice));
    IMG2D_CUDA(cudaMemcpy(dS, shot_fs, p->wave_elems * sizeof(cpx), cudaMemcpyHostToDevice));
    if ((rc = set_model(p, dO, dV, dk, dTF, dTB, 0))) return rc;
    MigrateArgs a = base_args(p, dW, dS);
    if ((rc = launch(p, a, dI, dIS, (long long)plane, 0))) return rc;
    IMG2D_CUDA(cudaDeviceSynchronize());
    if ((rc = read_status(p, 0))) return rc;
    if (image) IMG2D_CUDA(cudaMemcpy(image, dI, (size_t)nextrap * nx * sizeof(float), cudaMemcpyDeviceToHost));
    if (image_shots)
        IMG2D_CUDA(cudaMemcpy2D(image_shots, plane * sizeof(float), dIS, plane * sizeof(float),
                                (size_t)nextrap * nx * sizeof(float), ns, cudaMemcpyDeviceToHost));
    IMG2D_CUDA(cudaMemcpy(wave_fs, dW, p->wave_elems * sizeof(cpx), cudaMemcpyDeviceToHost));
    IMG2D_CUDA(cudaMemcpy(shot_fs, dS, p->wave_elems * sizeof(cpx), cudaMemcpyDeviceToHost));
    return IMG2D_OK;
}

}  // extern "C"
