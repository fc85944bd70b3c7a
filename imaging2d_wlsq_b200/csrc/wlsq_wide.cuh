// Wide cluster kernel: the decomposition of migrate_cluster2_kernel (wlsq_cluster2.cuh) reshaped so
// that a 2048-wide window needs a cluster of 2 CTAs instead of 4.
//
// Why: one CTA per SM holds one share of an item for the whole depth loop.  Clusters of 4 fit 33
// times on the 148 SMs of a B200 (132 SMs busy, because clusters cannot span GPCs), clusters of 2
// fit 74 times (all 148).  Each CTA here owns 1024 consecutive positions of 8 lane slots instead of
// 512 positions of 16 slots: the same 8192 (slot, position) pairs, the same shared memory for the
// wavefields, the same per-lane work (2 slots x 8 outputs) and the same operator reuse per load
// (each 16-byte tap pair feeds 2 taps x 2 slots x (S, conj R) = 32 FMAs of one lane).  An item
// carries 8 slots (one frequency), so there are twice as many items, each half as tall.
//
// Layout.  Lane group = 4 lanes; lane q holds slots q and q+4 of the item; 8 groups per warp, each
// over a block of X = 8 consecutive positions; 16 warps.  The wavefields of a position are 128
// bytes: for each lane q two float4, A = (S_a.re, S_b.re, S_a.im, S_b.im) and B = the same of
// conj(R) (a = slot q, b = slot q+4), so the two slots of a lane form the (x, y) halves of packed
// pairs.  The 8 groups of a warp read rows 8 positions apart, which without care would all hit
// banks 0-15; the A and B columns of a row are therefore swapped in every other 8-row block
// (column 2q + (h ^ ((pos >> 3) & 1)) for half h), so each bank serves 4 of the 32 lanes and a
// warp's 512-byte read takes the minimum 4 wavefronts.
//
// Arithmetic (per input t, output jj, tap (fr, fi)), for each of A and B:
//   re.ab += fr * v.re.ab ; re.ab += -fi * v.im.ab ; im.ab += fr * v.im.ab ; im.ab += fi * v.re.ab
// in that order per element, which is the FMA sequence of every other kernel of this library
// (IMG2D_MAC8), so final wavefields are bit-identical to migrate_cluster2_kernel.  ARITH = 1 issues
// it as packed f32x2 FMAs (FFMA2: two lanes of work per instruction), ARITH = 0 as scalar FMAs.
//
// Operator taps reach the tap loop through the per-lane-group shared-memory ring of the cluster2
// ring variant, copied with 16-byte cp.async two to three tap-loop iterations before they are read.  The next depth step's operator
// indices and this step's Kahan partial-image values of those two positions reach the thread
// through a per-thread shared-memory stage filled by cp.async a step ahead (STAGE, where the
// shared memory allows), or are loaded into registers at the start of the step.  The BULK variant
// fills the same ring with 1-D bulk copies completing on per-warp transaction-count barriers.
//
// Per depth step: tap loop into registers; aperture mask; edge outputs pushed into the neighbour's
// halo staging (distributed shared memory, double-buffered by step parity); the next step's first tap
// pairs copied; in-place write; imaging (Re(S conj R), shuffle over the group's 4 lanes, Kahan update
// of the CTA's private partial row); halo copy.  Warps wait for their two neighbours only (DF, below).
//
// Measured on a B200 against barriers of the CTA and the cluster in every step (FMA pipe 53% busy, 64%
// now): 256 uneven shots of 2048 x 80, 128 frequencies, 35 taps 47.1 -> 43.1 ms; 64 shots of 4096 x 30,
// 64 frequencies, 55 taps 13.2 -> 12.1 ms.
//
// Eight lanes per group (LANES = 8) give the 16-slot shape, 16 slots x 512 positions per CTA: each
// operator row feeds twice the multiply-adds.  It is the default where its clusters fill the GPU: 32
// shots of 1024 x 60, 256 frequencies, 31 taps 6.65 ms with migrate_cluster2_kernel's scalar FMAs,
// 6.39 ms with packed ones, 5.78 ms without the barriers.
#pragma once
#include "wlsq_cluster2.cuh"

namespace img2d {

template <int LANES>
struct WideShapeQ {
    static constexpr int Q = LANES;        // lanes per position group
    static constexpr int G = 2 * Q;        // lane slots per item (two per lane)
    static constexpr int P = 32 / Q;       // position groups per warp
    static constexpr int NW = 16;          // warps per CTA
    static constexpr int X = 8;            // positions per block
    static constexpr int PC = NW * P * X;  // positions per CTA (1024)
    static constexpr int NG = NW * P;      // lane groups per CTA (128)
    static constexpr int RING = 8 * kRingSlots + 1;  // float4 per lane group's ring (+1 pad)
};
typedef WideShapeQ<4> WideShape;
typedef WideShapeQ<8> Wide16Shape;

// Shared memory: ext[PC + 2 MP] rows + staging[2 parity][2 side][MP] rows (8 float4 per row) +
// the operator-pair rings.
template <class S = WideShape>
__host__ __device__ inline size_t wide_smem_bytes(int M)
{
    const int mp = cluster2_mp(M);
    return (size_t)((S::PC + 2 * mp) + 4 * mp) * S::G * 16 + (size_t)S::NG * S::RING * 16;
}

// Step-ahead stage (STAGE): per thread 6 words after the rings, the aligned index words holding the
// next depth step's operator indices of its two outputs and this step's Kahan partial and
// compensation values of its two positions.  Each thread reads only its own words, then refills
// them with cp.async for a later step.
template <class S = WideShape>
__host__ __device__ constexpr int wide_stage_words() { return 3 * (S::X / S::Q); }
template <class S = WideShape>
__host__ __device__ inline size_t wide_stage_smem_bytes(int M)
{
    return wide_smem_bytes<S>(M) + (size_t)S::NW * 32 * wide_stage_words<S>() * 4;
}

// BULK: two transaction-count barriers per warp after the stage words (or the rings), one per
// alternate ring chunk.
__host__ __device__ inline size_t wide_bulk_bar_offset(int M, bool stage)
{
    return stage ? wide_stage_smem_bytes(M) : wide_smem_bytes(M);
}
__host__ __device__ inline size_t wide_bulk_smem_bytes(int M, bool stage)
{
    return wide_bulk_bar_offset(M, stage) + (size_t)WideShape::NW * 2 * sizeof(unsigned long long);
}

// SM clock cycles (1.1 s) after which a ring-chunk wait gives up (waits for neighbours allow twice as
// many): the thread then records
// the failure in the plan's status word and neither waits for nor issues ring chunks again, so a
// phase that can never complete ends the launch instead of hanging it.
constexpr long long kBulkWaitCycles = 1ll << 31;

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

// the initialisations above become visible to the asynchronous (bulk-copy) proxy
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

// arrive on the barrier's current phase, first raising its expected transaction bytes
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long *bar, unsigned bytes)
{
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(
                     smem_addr(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity)
{
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return done != 0;
}

// plain arrival (release) on a barrier of this CTA
__device__ __forceinline__ void mbar_arrive(unsigned long long *bar)
{
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_addr(bar)) : "memory");
}

// arrival on a barrier of another CTA of the cluster (address from map_rank), releasing at cluster
// scope what this thread (and, after a __syncwarp, its warp) wrote there
__device__ __forceinline__ void mbar_arrive_cluster(unsigned addr)
{
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait_cluster(unsigned long long *bar, unsigned parity)
{
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return done != 0;
}

// 1-D bulk copy global -> this CTA's shared memory, completing bytes on the barrier (no multicast)
__device__ __forceinline__ void bulk_copy_g2s(void *dst, const void *src, unsigned bytes, unsigned long long *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

// float4 column of half h (0 = S, 1 = conj R) of lane q in row pos
template <int Q>
__device__ __forceinline__ int wide_col(int pos, int q, int h)
{
    return Q == 8 ? q + 8 * h : 2 * q + (h ^ ((pos >> 3) & 1));
}

template <int ARITH>
__device__ __forceinline__ void wide_mac(float (&c)[8], float fr, float fi, const float4 &va, const float4 &vb)
{
    if (ARITH == 1) {
        const float2 frr = make_float2(fr, fr), nfi = make_float2(-fi, -fi), fii = make_float2(fi, fi);
        float2 *c2 = reinterpret_cast<float2 *>(c);
        c2[0] = __ffma2_rn(frr, make_float2(va.x, va.y), c2[0]);
        c2[0] = __ffma2_rn(nfi, make_float2(va.z, va.w), c2[0]);
        c2[1] = __ffma2_rn(frr, make_float2(va.z, va.w), c2[1]);
        c2[1] = __ffma2_rn(fii, make_float2(va.x, va.y), c2[1]);
        c2[2] = __ffma2_rn(frr, make_float2(vb.x, vb.y), c2[2]);
        c2[2] = __ffma2_rn(nfi, make_float2(vb.z, vb.w), c2[2]);
        c2[3] = __ffma2_rn(frr, make_float2(vb.z, vb.w), c2[3]);
        c2[3] = __ffma2_rn(fii, make_float2(vb.x, vb.y), c2[3]);
    } else {
        c[0] = fmaf(fr, va.x, c[0]); c[0] = fmaf(-fi, va.z, c[0]);
        c[1] = fmaf(fr, va.y, c[1]); c[1] = fmaf(-fi, va.w, c[1]);
        c[2] = fmaf(fr, va.z, c[2]); c[2] = fmaf(fi, va.x, c[2]);
        c[3] = fmaf(fr, va.w, c[3]); c[3] = fmaf(fi, va.y, c[3]);
        c[4] = fmaf(fr, vb.x, c[4]); c[4] = fmaf(-fi, vb.z, c[4]);
        c[5] = fmaf(fr, vb.y, c[5]); c[5] = fmaf(-fi, vb.w, c[5]);
        c[6] = fmaf(fr, vb.z, c[6]); c[6] = fmaf(fi, vb.x, c[6]);
        c[7] = fmaf(fr, vb.w, c[7]); c[7] = fmaf(fi, vb.y, c[7]);
    }
}

// STAGE: the next step's operator indices and this step's Kahan values reach the thread through its
// shared-memory stage words, copied by cp.async one step ahead (no register holds a pending load
// across the tap loop); otherwise they are loaded into registers at the start of the step.
//
// BULK: the operator-pair ring is filled by 1-D bulk copies (cp.async.bulk, the copy engine of
// the SM) instead of per-lane 16-byte cp.async.  Ring iterations are copied in chunks of two (v
// even: the slots of v and v + 1 are adjacent), one bulk copy of up to 32 bytes per output, each
// chunk completing on one of two transaction-count barriers of the warp (alternating), where the
// cp.async ring would wait for a commit group.  A chunk is issued where the cp.async ring copies
// its later iteration and waited for where the ring waits for its first one.
//
// DF: no barrier of the CTA or the cluster inside the depth loop.  A warp's outputs need only its
// neighbours' rows (M <= the 8 P positions of a warp), so it waits for those two warps alone: before
// writing its rows in place, until they have read step l (barrier rd of the warp, two arrivals), and
// before reading step l + 1, until they have written theirs (wr).  At the edges of the CTA the pushed
// halo and an arrival from the neighbouring CTA's edge warp (hb) take the place of the neighbour; the
// edge warp copies the halo from the staging itself.  The staging of a parity is pushed again only
// after the pusher has received this CTA's push of the step between, which follows the copy; a pusher
// may be one step ahead, so even and odd exchanges have a barrier each.  rd and wr need only one: a
// neighbour's next arrival follows what this warp does after its wait.  With
// barriers every warp does its step-boundary work (writes, imaging, copies: a quarter of the step) at
// the same time and the FMA pipe idles; this way the warps of an SM sub-partition drift apart and one's
// boundary work runs beside the others' tap loops.  Every wait has a limit, like BULK's.
template <int ARITH, bool STAGE, bool BULK = false, int LANES = 4, bool DF = false>
__global__ void __launch_bounds__(WideShapeQ<LANES>::NW * 32, 1) migrate_wide_kernel(MigrateArgs a)
{
    using S = WideShapeQ<LANES>;
    constexpr int Q = S::Q, G = S::G, P = S::P, X = S::X, PC = S::PC;
    constexpr int NO = X / Q;  // outputs whose operator row, index and Kahan values a lane looks after
    constexpr int SW = wide_stage_words<S>();
    static_assert(!BULK || (Q == 4 && !DF), "the bulk-copy ring is built on 4 lanes per group and CTA barriers");
    const int M = a.M, L = 2 * a.M + 1;
    const int MP = cluster2_mp(M);
    const int NEXT = PC + 2 * MP;
    extern __shared__ float4 smem[];
    float4 *ext = smem;                     // [NEXT][G]; local position x at row x + MP
    float4 *stg = smem + (size_t)NEXT * G;  // [parity][side][MP][G]; side 0 = left halo, 1 = right
    float *extf = reinterpret_cast<float *>(ext);
    __shared__ int s_item;

    const unsigned crank = cluster_rank(), csize = cluster_size();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int p = lane / Q, q = lane % Q;
    const int b = warp * P + p;  // this lane group's block: local positions [b*X, b*X+X)
    // this lane group's ring, [output][slot] float4 plus one pad, after the halo staging
    float4 *const ringb = smem + (size_t)(NEXT + 4 * MP) * G + (size_t)b * S::RING;
    // STAGE: this thread's words [index word of each of its outputs q + o Q, then s and c of each]
    unsigned *const sst = reinterpret_cast<unsigned *>(smem + (size_t)(NEXT + 4 * MP) * G + (size_t)S::NG * S::RING) +
                          (size_t)threadIdx.x * SW;
    const int npairs = (L + 1) >> 1;
    static_assert(X == 8 && kRingSlots == 4, "the ring schedule assumes 8 outputs per block and 4 slots");
    // BULK: this warp's two chunk barriers, the chunks it has issued and waited for (warp-uniform)
    unsigned long long *const wbar =
        reinterpret_cast<unsigned long long *>(reinterpret_cast<char *>(smem) + wide_bulk_bar_offset(M, STAGE)) +
        warp * 2;
    unsigned n_issued = 0, n_waited = 0;
    bool bulk_failed = false;
    if (BULK) {
        if (lane == 0) {
            mbar_init(wbar, 32);  // one arrival per lane and chunk
            mbar_init(wbar + 1, 32);
            mbar_init_fence();
        }
        __syncwarp();
    }
    // DF: barriers of each warp and of the two edges, the phases this warp has waited for
    __shared__ unsigned long long s_rd[DF ? S::NW : 1], s_wr[DF ? S::NW : 1], s_hb[4];
    unsigned n_rd = 0, n_wr = 0, hb_base = 0;
    bool wait_failed = false;
    if (DF && threadIdx.x < S::NW) {
        mbar_init(s_rd + threadIdx.x, 2);
        mbar_init(s_wr + threadIdx.x, 2);
        if (threadIdx.x < 4) mbar_init(s_hb + threadIdx.x, 1);
        mbar_init_fence();  // made visible to the cluster by the first item's barriers
    }
    auto df_wait = [&](unsigned long long *bar, unsigned phase, bool cluster) {
        auto ready = [&]() { return cluster ? mbar_try_wait_cluster(bar, phase & 1) : mbar_try_wait(bar, phase & 1); };
        if (wait_failed || ready()) return;
        const long long t0 = clock64();
        while (!ready()) {
            if (clock64() - t0 > 2 * kBulkWaitCycles) {
                wait_failed = true;
                if (a.status) atomicOr(a.status, 2);
                break;
            }
        }
    };
    const unsigned rank0_item = map_rank(&s_item, 0);
    const int row_bytes = a.tab_stride * 8;
    // register budget (512 threads at <= 128 registers): the partial-image, table and owner
    // pointers are formed from the kernel parameters where they are used

    for (;;) {
        if (crank == 0 && threadIdx.x == 0) s_item = atomicAdd(a.counter, 1);
        cluster_arrive();
        cluster_wait();
        const int it = ld_cluster_s32(rank0_item);
        cluster_arrive();
        cluster_wait();
        if (it >= a.n_items) break;
        const int2 item = a.items[it];
        const GroupDesc grp = a.groups[item.x];
        const int j = item.y, u0 = grp.u0, W = grp.W;
        // The item's window is split evenly over the cluster in units of 4 warps (256 positions, one
        // warp per SM sub-partition): each CTA owns NC <= PC consecutive positions starting at c0,
        // and warps past NC skip the step's work.  A narrow window then leaves every sub-partition
        // one warp less to run instead of computing positions past the window (finer units would
        // leave the busiest sub-partition as loaded as before).
        const int NC = min(PC, (W + (int)csize * 256 - 1) / ((int)csize * 256) * 256);
        const int c0 = (int)crank * NC;
        const int own = max(0, min(NC, W - c0));  // window positions this CTA owns (the rest are past W)
        const bool warp_active = warp * (P * X) < NC;
        const bool push_left = crank > 0 && b * X < MP;
        const bool push_right = crank + 1 < csize && b * X + X > NC - MP && b * X < NC;

        for (int i = threadIdx.x; i < (NEXT + 4 * MP) * G; i += blockDim.x) smem[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncthreads();
        for (int k = grp.seg_begin; k < grp.seg_begin + grp.nseg; ++k) {
            const int4 sg = a.segs[k];
            const int r0 = sg.z - u0;
            const int lo = max(r0, c0 - MP), hi = min(r0 + sg.w, c0 + NC + MP);
            const cpx *ws = a.wave + a.shot_off[sg.x] + (long long)j * sg.w;
            const cpx *rs = a.shot + a.shot_off[sg.x] + (long long)j * sg.w;
            const int sq = sg.y & (Q - 1), sh = sg.y / Q;  // lane and half (x/z or y/w) of the slot
            for (int x = lo + (int)threadIdx.x; x < hi; x += blockDim.x) {
                const cpx Sv = ws[x - r0], Rv = rs[x - r0];
                const int pos = x - c0 + MP;
                float *fa = extf + ((size_t)pos * G + wide_col<Q>(pos, sq, 0)) * 4;
                float *fb = extf + ((size_t)pos * G + wide_col<Q>(pos, sq, 1)) * 4;
                fa[sh] = Sv.re;
                fa[2 + sh] = Sv.im;
                fb[sh] = Rv.re;
                fb[2 + sh] = -Rv.im;
            }
        }
        // cluster-wide: no CTA may push step-0 halos into a peer that is still zeroing them
        cluster_arrive();
        cluster_wait();

        const bool blk_active = b * X < own;
        unsigned in_a = 0, in_b = 0;  // bit jj: output jj of slot q (q+4) is inside a shot's aperture
        {
            const int16_t *own_a = (blk_active && q < grp.nslots)
                                       ? a.owner + grp.owner_off + (long long)q * grp.owner_stride + c0 + b * X
                                       : nullptr;
            const int16_t *own_b = (blk_active && q + Q < grp.nslots)
                                       ? a.owner + grp.owner_off + (long long)(q + Q) * grp.owner_stride + c0 + b * X
                                       : nullptr;
            int16_t oa[X], ob[X];
            load_owner<X>(own_a, oa);
            load_owner<X>(own_b, ob);
#pragma unroll
            for (int jj = 0; jj < X; ++jj) {
                in_a |= (oa[jj] >= 0 ? 1u : 0u) << jj;
                in_b |= (ob[jj] >= 0 ? 1u : 0u) << jj;
            }
        }
        const uint16_t *idx_j = a.idx + (long long)j * a.idx_jstride;
        const int xg = u0 + c0 + b * X;  // model position of the block's first output
        // lane q owns outputs q + o Q of the block: their operator rows (byte offsets into the table),
        // next-step indices and Kahan partial-image values
        int xq[NO];
        bool imgo[NO];
        unsigned roff[NO];
        unsigned nidx = 0;  // next step's row indices of the lane's outputs (16 bits each)
#pragma unroll
        for (int o = 0; o < NO; ++o) {
            xq[o] = min(xg + q + o * Q, a.nx - 1);
            imgo[o] = a.partial && b * X + q + o * Q < own;
            roff[o] = (unsigned)idx_j[xq[o]] * (unsigned)row_bytes;
        }
        // STAGE: copies of the aligned index words of step ls and of the Kahan values of step lk into
        // this thread's stage words
        auto stage_idx = [&](int ls) {
            const uint16_t *ip = idx_j + (long long)ls * a.idx_lstride;
#pragma unroll
            for (int o = 0; o < NO; ++o) cp_async4(sst + o, ip + (xq[o] & ~1));
        };
        const long long prow0 = (long long)blockIdx.x * a.nextrap * a.nx + xg + q;  // partial element of step 0
        auto stage_kahan = [&](int lk) {
            const long long e = prow0 + (long long)lk * a.nx;
#pragma unroll
            for (int o = 0; o < NO; ++o)
                if (imgo[o]) {
                    cp_async4(sst + NO + 2 * o, a.partial + e + o * Q);
                    cp_async4(sst + NO + 2 * o + 1, a.comp + e + o * Q);
                }
        };
        // Ring copies go in chunks of two iterations (v even, v and v + 1), whose pairs are 32
        // consecutive bytes of a row: two lanes copy one output's 32 bytes, so a copy instruction of
        // the warp touches 16 cache lines.  One lane per output and 16 bytes touched 32, and the L1 tag
        // lookups, one line a cycle, took as long as the multiply-adds they fed (leaving the copies out
        // altogether: 12% on the uneven survey).  rcopy[i]: the rows this lane copies from.
        constexpr int NCP = X * 2 / Q;  // copies per lane and chunk
        const int rh = q & 1;
        unsigned rcopy[NCP];
        auto spread_rows = [&]() {
#pragma unroll
            for (int i = 0; i < NCP; ++i) {
                // output of copy i: (q >> 1) + i Q / 2, owned by lane (output mod Q) of the group
                const int o = i * (Q / 2) / Q;
                rcopy[i] = __shfl_sync(0xffffffffu, roff[o], ((q >> 1) + i * (Q / 2)) & (Q - 1), Q);
            }
        };
        auto ring_pair = [&](int v, bool both) {
            const char *tabb = reinterpret_cast<const char *>(a.tabF);
            if (!both && rh) return;
            const int sl = (v + rh) & (kRingSlots - 1);
#pragma unroll
            for (int i = 0; i < NCP; ++i) {
                const int o = (q >> 1) + i * (Q / 2);
                const int pr = v + rh + ((X - o) >> 1);
                const bool ok = (unsigned)pr < (unsigned)npairs;
                // branch-free: a pair outside the row becomes a zero-filled copy of nothing (never read)
                cp_async16_zfill(ringb + o * kRingSlots + sl, tabb + rcopy[i] + (ok ? pr : 0) * 16, ok ? 16u : 0u);
            }
        };
        // BULK: the pairs of ring iterations v and v + 1 (v even; v + 1 only while <= vlast) of outputs
        // q and q + 4, one bulk copy per output into the two adjacent slots.  Pairs outside the row
        // are not copied (their slots are never read).  Every lane arrives on the chunk's barrier
        // with its own byte count before issuing its copies, so the phase completes only after all
        // 32 lanes' copies have landed.
        auto ring_chunk = [&](int v, int vlast) {
            const char *tabb = reinterpret_cast<const char *>(a.tabF);
            unsigned long long *bar = wbar + (n_issued & 1);
            ++n_issued;
            if (bulk_failed) return;  // never arrive on a phase that may still be open
            unsigned nb[2];
            const char *src[2];
            float4 *dst[2];
#pragma unroll
            for (int o = 0; o < 2; ++o) {
                const int p0 = v + ((X - q - o * Q) >> 1);
                const bool ok0 = (unsigned)p0 < (unsigned)npairs;
                const bool ok1 = v + 1 <= vlast && (unsigned)(p0 + 1) < (unsigned)npairs;
                const int first = ok0 ? 0 : 1;
                nb[o] = (ok0 ? 16u : 0u) + (ok1 ? 16u : 0u);
                src[o] = tabb + roff[o < NO ? o : 0] + (long long)(p0 + first) * 16;
                dst[o] = ringb + (q + o * Q) * kRingSlots + (v & (kRingSlots - 1)) + first;
            }
            mbar_arrive_expect_tx(bar, nb[0] + nb[1]);
            if (nb[0]) bulk_copy_g2s(dst[0], src[0], nb[0], bar);
            if (nb[1]) bulk_copy_g2s(dst[1], src[1], nb[1], bar);
        };
        // BULK: wait for the oldest chunk not yet waited for (chunks are waited for in issue order,
        // and a barrier's next chunk is issued only after its previous one was waited for)
        auto chunk_wait = [&]() {
            unsigned long long *bar = wbar + (n_waited & 1);
            const unsigned parity = (n_waited >> 1) & 1;
            ++n_waited;
            if (bulk_failed || mbar_try_wait(bar, parity)) return;
            const long long t0 = clock64();
            while (!mbar_try_wait(bar, parity)) {
                if (clock64() - t0 > kBulkWaitCycles) {
                    bulk_failed = true;
                    if (a.status) atomicOr(a.status, 1);
                    break;
                }
            }
        };
        if (warp_active) {
            if (BULK) {
                ring_chunk(-4, -1);
                ring_chunk(-2, -1);
            } else {
                spread_rows();
                ring_pair(-4, true);
                ring_pair(-2, true);
            }
            if (STAGE) {
                if (a.nextrap > 1) stage_idx(1);
                stage_kahan(0);
            }
        }
        cp_async_commit();
        // DF: the warps whose rows this one shares (itself where there is none: the barriers expect two)
        const int last_warp = NC / (P * X) - 1;
        const int wl = max(warp - 1, 0), wr = min(warp + 1, last_warp);
        const bool hb_left = DF && warp == 0 && crank > 0, hb_right = DF && warp == last_warp && crank + 1 < csize;
        auto df_signal = [&](unsigned long long *bars) {
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(bars + wl);
                mbar_arrive(bars + wr);
            }
        };
        const int srow0 = b * X + MP - M;  // row of input t = 0
        const int nmid = (L - X + 1) / 2;  // middle tap-loop iterations (two inputs each)

        for (int l = 0; l < a.nextrap && (!DF || warp_active); ++l) {
            const int par = l & 1;
            if (DF && l > 0) {
                // the neighbours' rows of this step, or the halo pushed by the neighbouring CTA
                df_wait(s_wr + warp, n_wr++, false);
                if (hb_left || hb_right) {
                    const unsigned ex = hb_base + l - 1;  // exchange number: its barriers, their phase
                    const float4 *hs = stg + (size_t)(par * 2) * MP * G;
                    if (hb_left) {
                        df_wait(s_hb + (ex & 1), ex >> 1, true);
                        for (int i = lane; i < MP * G; i += 32) ext[i] = hs[i];
                    }
                    if (hb_right) {
                        df_wait(s_hb + 2 + (ex & 1), ex >> 1, true);
                        for (int i = lane; i < MP * G; i += 32) ext[(NC + MP) * G + i] = hs[MP * G + i];
                    }
                    __syncwarp();
                }
            }
            // this step's prologue pairs (copied at the end of the previous step) for the group
            cp_async_wait_all();
            if (BULK && warp_active) {
                chunk_wait();
                chunk_wait();
            }
            __syncwarp();  // control flow is warp-uniform here
            const long long pe = prow0 + (long long)l * a.nx;
            float cur_s[NO] = {}, cur_c[NO] = {};
            if (!STAGE) {
                // this step's Kahan values and the next step's operator indices: the loads are
                // issued here and complete during the tap loop
#pragma unroll
                for (int o = 0; o < NO; ++o)
                    if (imgo[o]) {
                        cur_s[o] = a.partial[pe + o * Q];
                        cur_c[o] = a.comp[pe + o * Q];
                    }
                if (l + 1 < a.nextrap) {
                    const uint16_t *inext = idx_j + (long long)(l + 1) * a.idx_lstride;
                    nidx = 0;
#pragma unroll
                    for (int o = 0; o < NO; ++o) nidx |= (unsigned)inext[xq[o]] << (16 * o);
                }
            }
            // the partial-image rows of the next step into L2 (read at the end of this step by the
            // stage, or at the start of the next one)
            if (q == 0 && imgo[0] && l + 1 < a.nextrap) {
                asm volatile("prefetch.global.L2 [%0];" ::"l"(a.partial + pe + a.nx));
                asm volatile("prefetch.global.L2 [%0];" ::"l"(a.comp + pe + a.nx));
            }
            float acc[X][8];
#pragma unroll
            for (int jj = 0; jj < X; ++jj)
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[jj][e] = 0.f;
            if (warp_active) {  // warps past the CTA's share of the window skip the step's work
            float4 tp[X];
            // input t: row srow0 + t, columns wide_col<Q>(row, q, 0/1)
            auto load_in = [&](int row, float4 &va, float4 &vb) {
                if (Q == 8) {
                    const float4 *r = ext + (size_t)row * G + q;
                    va = r[0];
                    vb = r[8];
                } else {
                    const float4 *r = ext + (size_t)row * G + 2 * q;
                    const int sw = (row >> 3) & 1;
                    va = r[sw];
                    vb = r[sw ^ 1];
                }
            };

            // prologue: t = 0 .. X-2, outputs jj <= t are active
#pragma unroll
            for (int t = 0; t < X - 1; ++t) {
                float4 va, vb;
                load_in(srow0 + t, va, vb);
#pragma unroll
                for (int jj = 0; jj < X; ++jj) {
                    const int k = t - jj;
                    if (k >= 0) {
                        if ((k & 1) == 0)
                            tp[jj] = ringb[jj * kRingSlots + (((k >> 1) - ((X - jj) >> 1)) & (kRingSlots - 1))];
                        const float fr = (k & 1) ? tp[jj].z : tp[jj].x;
                        const float fi = (k & 1) ? tp[jj].w : tp[jj].y;
                        wide_mac<ARITH>(acc[jj], fr, fi, va, vb);
                    }
                }
                // the slots of iterations -4 and -3 have been read: copy iterations 0 and 1
                if (t == 2) {
                    if (BULK) {
                        ring_chunk(0, nmid + 3);
                    } else {
                        ring_pair(0, true);
                        cp_async_commit();
                    }
                }
            }
            // middle: t = X-1 .. L-1 in steps of two (odd t, then even t+1)
            int row = srow0 + X - 1;
            for (int u = 0; u < nmid; ++u, row += 2) {
                const float4 *rs = ringb + (u & (kRingSlots - 1));
                // iterations u - 2 and u - 1 have read the slots of u + 2 and u + 3; wait for u and u + 1
                if (!(u & 1)) {
                    if (BULK) {
                        ring_chunk(u + 2, nmid + 3);
                        chunk_wait();
                    } else {
                        ring_pair(u + 2, true);
                        cp_async_commit();
                        cp_async_wait<1>();
                    }
                    __syncwarp();  // control flow is warp-uniform here
                }
                {
                    float4 va, vb;
                    load_in(row, va, vb);
#pragma unroll
                    for (int jj = 0; jj < X; ++jj) {
                        if (jj & 1) tp[jj] = rs[jj * kRingSlots];
                        const float fr = (jj & 1) ? tp[jj].x : tp[jj].z;
                        const float fi = (jj & 1) ? tp[jj].y : tp[jj].w;
                        wide_mac<ARITH>(acc[jj], fr, fi, va, vb);
                    }
                }
                {
                    float4 va, vb;
                    load_in(row + 1, va, vb);
#pragma unroll
                    for (int jj = 0; jj < X; ++jj) {
                        if (!(jj & 1)) tp[jj] = rs[jj * kRingSlots];
                        const float fr = (jj & 1) ? tp[jj].z : tp[jj].x;
                        const float fi = (jj & 1) ? tp[jj].w : tp[jj].y;
                        wide_mac<ARITH>(acc[jj], fr, fi, va, vb);
                    }
                }
            }
            // epilogue: t = L .. L+X-2, outputs jj > t-L are active (k = t - jj <= L-1)
            if (BULK) {
                ring_chunk((nmid + 3) & ~1, nmid + 3);
            } else {
                // for odd nmid iteration nmid + 4, whose slot iteration nmid has yet to read, does not exist
                ring_pair((nmid + 3) & ~1, !(nmid & 1));
                cp_async_commit();
            }
#pragma unroll
            for (int e = 0; e < X - 1; ++e) {
                float4 va, vb;
                load_in(srow0 + L + e, va, vb);
                // steps e and e + 1 read iteration nmid + e / 2; the last two chunks may be in flight
                if ((e & 1) == 0 && !((nmid + (e >> 1)) & 1)) {
                    if (BULK) chunk_wait();
                    else if (e < 4) cp_async_wait<1>();
                    else cp_async_wait<0>();
                    __syncwarp();  // control flow is warp-uniform here
                }
#pragma unroll
                for (int jj = 0; jj < X; ++jj) {
                    if (jj > e) {
                        // k = L + e - jj, parity of (1 + e - jj) since L is odd
                        const bool even = ((1 + e - jj) & 1) == 0;
                        if (even) tp[jj] = ringb[jj * kRingSlots + ((nmid + (e >> 1)) & (kRingSlots - 1))];
                        const float fr = even ? tp[jj].x : tp[jj].z;
                        const float fi = even ? tp[jj].y : tp[jj].w;
                        wide_mac<ARITH>(acc[jj], fr, fi, va, vb);
                    }
                }
            }
            if (DF) df_signal(s_rd);  // this warp has read its neighbours' rows of step l
            // outputs outside every shot aperture of their slot stay zero; most lanes have none
            if ((in_a & in_b) != (1u << X) - 1u) {
#pragma unroll
                for (int jj = 0; jj < X; ++jj) {
                    if (!((in_a >> jj) & 1u)) acc[jj][0] = acc[jj][2] = acc[jj][4] = acc[jj][6] = 0.f;
                    if (!((in_b >> jj) & 1u)) acc[jj][1] = acc[jj][3] = acc[jj][5] = acc[jj][7] = 0.f;
                }
            }
            // halos of step l+1 into the neighbours' staging (parity par^1): left neighbour's right
            // halo rows are its ext rows PC + MP + x, right neighbour's left halo rows its rows x
            if (push_left) {
                float4 *dst = stg + ((size_t)((par ^ 1) * 2 + 1) * MP) * G;
#pragma unroll
                for (int jj = 0; jj < X; ++jj) {
                    const int x = b * X + jj;
                    if (x < MP) {
                        const int prow = NC + MP + x;
                        const unsigned ra = map_rank(dst + (size_t)x * G, crank - 1);
                        st_cluster(ra + wide_col<Q>(prow, q, 0) * 16, make_float4(acc[jj][0], acc[jj][1], acc[jj][2], acc[jj][3]));
                        st_cluster(ra + wide_col<Q>(prow, q, 1) * 16, make_float4(acc[jj][4], acc[jj][5], acc[jj][6], acc[jj][7]));
                    }
                }
            }
            if (push_right) {
                float4 *dst = stg + ((size_t)((par ^ 1) * 2 + 0) * MP) * G;
#pragma unroll
                for (int jj = 0; jj < X; ++jj) {
                    const int x = b * X + jj - (NC - MP);
                    if (x >= 0) {
                        const unsigned ra = map_rank(dst + (size_t)x * G, crank + 1);
                        st_cluster(ra + wide_col<Q>(x, q, 0) * 16, make_float4(acc[jj][0], acc[jj][1], acc[jj][2], acc[jj][3]));
                        st_cluster(ra + wide_col<Q>(x, q, 1) * 16, make_float4(acc[jj][4], acc[jj][5], acc[jj][6], acc[jj][7]));
                    }
                }
            }
            if (DF && l + 1 < a.nextrap && (hb_left || hb_right)) {
                __syncwarp();
                // the right edge of the CTA to the left, the left edge of the CTA to the right
                if (lane == 0) {
                    if (hb_left) mbar_arrive_cluster(map_rank(s_hb + 2 + ((hb_base + l) & 1), crank - 1));
                    if (hb_right) mbar_arrive_cluster(map_rank(s_hb + ((hb_base + l) & 1), crank + 1));
                }
            }
            }  // warp_active
            // The neighbours read only their halo staging (the pushes above), never this CTA's ext[]:
            // arrive now, so the barrier's release covers the pushes but not the in-place writes.
            // The staging of parity par^1 is rewritten (step l+2) only after this CTA's arrival of
            // step l+1, which follows its copy of that staging at the end of this step.
            if (!DF) cluster_arrive();
            // every ring slot has been read: copy the next step's prologue pairs (u < 0) now, so
            // that they arrive during the halo exchange and the imaging
            if (warp_active && l + 1 < a.nextrap) {
#pragma unroll
                for (int o = 0; o < NO; ++o)
                    roff[o] = (STAGE ? (sst[o] >> (16 * (xq[o] & 1))) & 0xffffu : (nidx >> (16 * o)) & 0xffffu) *
                              (unsigned)row_bytes;
                if (BULK) {
                    ring_chunk(-4, -1);
                    ring_chunk(-2, -1);
                } else {
                    spread_rows();
                    ring_pair(-4, true);
                    ring_pair(-2, true);
                }
                // the words just read are refilled for step l + 2 (their reads are complete: the
                // copies above used them)
                if (STAGE && l + 2 < a.nextrap) stage_idx(l + 2);
            }
            cp_async_commit();
            // in place, once every read of step l's values in this warp's rows of ext[] is done
            auto write_rows = [&]() {
#pragma unroll
                for (int jj = 0; jj < X; ++jj) {
                    const int prow = b * X + MP + jj;
                    float4 *dst = ext + (size_t)prow * G;
                    dst[wide_col<Q>(prow, q, 0)] = make_float4(acc[jj][0], acc[jj][1], acc[jj][2], acc[jj][3]);
                    dst[wide_col<Q>(prow, q, 1)] = make_float4(acc[jj][4], acc[jj][5], acc[jj][6], acc[jj][7]);
                }
            };
            if (DF) {
                df_wait(s_rd + warp, n_rd++, false);
                write_rows();
                if (l + 1 < a.nextrap) df_signal(s_wr);
            } else {
                __syncthreads();
            }
            if (warp_active) {
            if (!DF) write_rows();
            // Re(S conj R) of both slots per output, summed over the group's 4 lanes by a reduce-scatter:
            // exchange across lanes q ^ 2 keeps the 4 outputs with (jj & 2) == (q & 2), exchange
            // across q ^ 1 keeps jj = q and q + 4 (6 shuffles instead of 8 x 2)
            float img[X];
#pragma unroll
            for (int jj = 0; jj < X; ++jj) {
                const float ia = acc[jj][0] * acc[jj][4] - acc[jj][2] * acc[jj][6];
                const float ib = acc[jj][1] * acc[jj][5] - acc[jj][3] * acc[jj][7];
                if (a.image_shots) {
                    // per-shot images (optional output): shot ids re-read from the owner table
                    const GroupDesc &g2 = a.groups[item.x];
                    const int16_t *orow = a.owner + g2.owner_off + c0 + b * X + jj;
                    if ((in_a >> jj) & 1u)
                        atomicAdd(a.image_shots + (long long)orow[(long long)q * g2.owner_stride] * a.img_sstride +
                                      (long long)l * a.nx + xg + jj, ia);
                    if ((in_b >> jj) & 1u)
                        atomicAdd(a.image_shots + (long long)orow[(long long)(q + Q) * g2.owner_stride] * a.img_sstride +
                                      (long long)l * a.nx + xg + jj, ib);
                }
                img[jj] = ia + ib;
            }
            // a reduce-scatter: each exchange halves the outputs a lane keeps, until q + o Q are left
            float img_q[NO];
            if constexpr (Q == 8) {
                const bool hi4 = (q & 4) != 0, hi2 = (q & 2) != 0, hi1 = (q & 1) != 0;
                float r4[4], r2[2];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float keep = hi4 ? img[i + 4] : img[i], send = hi4 ? img[i] : img[i + 4];
                    r4[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float keep = hi2 ? r4[i + 2] : r4[i], send = hi2 ? r4[i] : r4[i + 2];
                    r2[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
                }
                const float keep = hi1 ? r2[1] : r2[0], send = hi1 ? r2[0] : r2[1];
                img_q[0] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
            } else {
                const bool hi2 = (q & 2) != 0, hi1 = (q & 1) != 0;
                float r4[4];  // outputs {0, 1, 4, 5} ^ (q & 2)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int base = (i & 1) | ((i & 2) << 1);
                    const float keep = hi2 ? img[base ^ 2] : img[base];
                    const float send = hi2 ? img[base] : img[base ^ 2];
                    r4[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
                }
#pragma unroll
                for (int k = 0; k < NO; ++k) {
                    const float keep = hi1 ? r4[2 * k + 1] : r4[2 * k];
                    const float send = hi1 ? r4[2 * k] : r4[2 * k + 1];
                    img_q[k] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
                }
            }
            // Kahan update (the operations of kahan_add) on the values loaded at the step's start
#pragma unroll
            for (int o = 0; o < NO; ++o) {
                if (STAGE) {
                    cur_s[o] = __uint_as_float(sst[NO + 2 * o]);
                    cur_c[o] = __uint_as_float(sst[NO + 2 * o + 1]);
                }
                if (imgo[o]) {
                    const float y = img_q[o] - cur_c[o];
                    const float t = cur_s[o] + y;
                    a.partial[pe + o * Q] = t;
                    a.comp[pe + o * Q] = (t - cur_s[o]) - y;
                }
            }
            if (STAGE && l + 1 < a.nextrap) stage_kahan(l + 1);  // refilled for the next step
            }  // warp_active
            if (STAGE) cp_async_commit();  // the Kahan words, waited for at the next step's start
            if (DF) continue;
            cluster_wait();
            const float4 *hs = stg + (size_t)((par ^ 1) * 2) * MP * G;
            for (int i = threadIdx.x; i < 2 * MP * G; i += blockDim.x) {
                const int side = i / (MP * G), r = i % (MP * G);
                ext[(side ? (NC + MP) * G : 0) + r] = hs[i];
            }
            __syncthreads();
        }
        if (DF) {
            hb_base += a.nextrap - 1;
            __syncthreads();  // every warp's rows of the last step are written
        }
        if (a.write_back) {
            for (int k = grp.seg_begin; k < grp.seg_begin + grp.nseg; ++k) {
                const int4 sg = a.segs[k];
                const int r0 = sg.z - u0;
                const int lo = max(r0, c0), hi = min(r0 + sg.w, c0 + own);
                cpx *ws = a.wave + a.shot_off[sg.x] + (long long)j * sg.w;
                cpx *rs = a.shot + a.shot_off[sg.x] + (long long)j * sg.w;
                const int sq = sg.y & (Q - 1), sh = sg.y / Q;
                for (int x = lo + (int)threadIdx.x; x < hi; x += blockDim.x) {
                    const int pos = x - c0 + MP;
                    const float *fa = extf + ((size_t)pos * G + wide_col<Q>(pos, sq, 0)) * 4;
                    const float *fb = extf + ((size_t)pos * G + wide_col<Q>(pos, sq, 1)) * 4;
                    ws[x - r0] = cpx{fa[sh], fa[2 + sh]};
                    rs[x - r0] = cpx{fb[sh], -fb[2 + sh]};
                }
            }
        }
        __syncthreads();
    }
    cluster_arrive();
    cluster_wait();
}

}  // namespace img2d
