// Demigration of surveys with at least 12 lane slots: the recursion, checkpoints and slabs of
// wlsq_adjoint.cuh on the migration's wide shape (wlsq_wide.cuh).
//
// One item = 16 lane slots x one frequency; its window is split over a cluster of CTAs of 1024
// positions.  A group of 4 lanes owns a block of 8 positions, lane q the slots q, q + 4, q + 8 and
// q + 12: a 16-byte tap pair feeds 2 taps x 4 slots = 32 multiply-adds of a lane, twice what two slots
// per lane gave (the kernel before: 8 lanes x 2 slots, 512 positions per CTA), and those loads are what
// a demigration step waits for.  A position is 128 bytes: per lane two float4, (re, im) of slots a, b
// as (a.re, b.re, a.im, b.im) and the same of c, d, so the multiply-adds are packed (FFMA2).
//
// The field is updated in place, as in the migration.  Every operation of the recursion (a forward
// step, a transposed step, a reload of a checkpoint or of the saved adjoint state) ends the same way:
// the warp says that it has read its neighbours' rows, pushes its edge rows into the neighbouring CTA's
// staging, waits until its neighbours have read, writes, and says so.  A warp waits for nobody else
// inside an item: positions, and with them all global planes, belong to one thread from end to end.
//
// Forward steps take their tap pairs through the migration's shared-memory ring.  Transposed steps read
// runs of 8 consecutive taps of each input position's row through L1; the row numbers of a warp's 64
// positions and both halos are kept in shared memory one step ahead.  Both run for any operator
// length.  The multiply-adds of an element come in the order of the single-CTA kernel: results are
// bit-identical.
//
// Measured on a B200: the demigration of 64 shots of 1024 x 500, 256 frequencies, 31 taps with kept
// checkpoints 196 -> 125 ms; lengths the kernel before ran without unrolling gain more (32 shots of
// 900 x 100, 96 frequencies, 47 taps, one least-squares gradient: 33.9 -> 15.8 ms).  FMA pipe 49% busy,
// issue 41%: what is left waits for the operator rows of the transposed step (L1 holds a quarter of
// them; prefetching them three inputs ahead cost 5%, the prefetches take the same L1 lookups).
#pragma once
#include "wlsq_adjoint.cuh"
#include "wlsq_wide.cuh"

namespace img2d {

struct DemigWideShape {
    static constexpr int Q = 4, P = 8, X = 8, NW = 16;
    static constexpr int G = 16;           // lane slots per item
    static constexpr int PC = NW * P * X;  // positions per CTA (1024)
    static constexpr int NG = NW * P;      // lane groups per CTA
    static constexpr int ROW = 8;          // float4 per position
    static constexpr int RING = 8 * kRingSlots + 1;
};

// Positions of a window of W per CTA of a cluster of K: an even split in whole warps (64 positions).  In
// units of 256, as the migration splits, a window of 300 ran 8 warps of which 5 had work.
__host__ __device__ inline int demigw_share(int W, int K) { return (W + K * 64 - 1) / (K * 64) * 64; }

// row numbers of a warp's 64 positions and MP more on either side
__host__ __device__ inline int demigw_idx(int M) { return 64 + 2 * cluster2_mp(M); }

__host__ __device__ inline size_t demigw_smem_bytes(int M)
{
    using S = DemigWideShape;
    const int mp = cluster2_mp(M);
    return (size_t)(S::PC + 2 * mp + 4 * mp) * S::ROW * 16 + (size_t)S::NG * S::RING * 16 +
           (size_t)S::NW * 2 * demigw_idx(M) * 2;
}

// RING: forward steps through the ring; else their taps come through L1 too.
template <bool RING>
__global__ void __launch_bounds__(DemigWideShape::NW * 32, 1) demigrate_wide_kernel(DemigrateArgs a, int *status)
{
    using S = DemigWideShape;
    constexpr int Q = S::Q, P = S::P, X = S::X, ROW = S::ROW;
    const int M = a.M, L = 2 * a.M + 1, MP = cluster2_mp(a.M);
    const int NEXT = S::PC + 2 * MP;
    extern __shared__ float4 smem[];
    float4 *ext = smem;                        // [NEXT][ROW]; local position x at row x + MP
    float4 *stg = smem + (size_t)NEXT * ROW;   // [parity][side][MP][ROW]
    __shared__ int s_item;
    __shared__ unsigned long long s_rd[S::NW], s_wr[S::NW], s_hb[4];

    const unsigned crank = cluster_rank(), csize = cluster_size();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int p = lane / Q, q = lane % Q;
    const int b = warp * P + p;
    float4 *const ringb = smem + (size_t)(NEXT + 4 * MP) * ROW + (size_t)b * S::RING;
    const int NI = demigw_idx(M);
    uint16_t *const idxw = reinterpret_cast<uint16_t *>(smem + (size_t)(NEXT + 4 * MP) * ROW + (size_t)S::NG * S::RING) +
                           (size_t)warp * 2 * NI;
    const int npairs = (L + 1) >> 1;
    const int row_bytes = a.tab_stride * 8;
    const char *tabb = reinterpret_cast<const char *>(a.tab);
    const unsigned rank0_item = map_rank(&s_item, 0);
    const long long pe = (long long)a.plane * ROW;  // float4 per plane
    float4 *work = reinterpret_cast<float4 *>(a.work) + (long long)blockIdx.x * (a.work_cta / 2);
    float4 *slabbuf = work + (long long)a.nslab * pe;
    float4 *save = slabbuf + (long long)a.slab * pe;
    const int D = a.slab;
    unsigned n_op = 0;      // operations of this warp (phases of its barriers)
    unsigned hb_base = 0;   // operations of the CTA's items before this one (phases of the edge barriers)
    bool wait_failed = false;

    if (threadIdx.x < S::NW) {
        mbar_init(s_rd + threadIdx.x, 2);
        mbar_init(s_wr + threadIdx.x, 2);
        if (threadIdx.x < 4) mbar_init(s_hb + threadIdx.x, 1);
        mbar_init_fence();
    }
    auto wait = [&](unsigned long long *bar, unsigned phase, bool cluster) {
        auto ready = [&]() { return cluster ? mbar_try_wait_cluster(bar, phase & 1) : mbar_try_wait(bar, phase & 1); };
        if (wait_failed || ready()) return;
        const long long t0 = clock64();
        while (!ready()) {
            if (clock64() - t0 > 2 * kBulkWaitCycles) {
                wait_failed = true;
                atomicOr(status, 2);
                break;
            }
        }
    };

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
        const int NC = demigw_share(W, (int)csize);
        const int c0 = (int)crank * NC;
        const int own = max(0, min(NC, W - c0));
        const bool warp_active = warp * (P * X) < NC;
        const int last_warp = NC / (P * X) - 1;
        const int wl = max(warp - 1, 0), wr = min(warp + 1, last_warp);
        const bool hb_left = warp == 0 && crank > 0, hb_right = warp == last_warp && crank + 1 < csize;
        const bool push_left = crank > 0 && b * X < MP;
        const bool push_right = crank + 1 < csize && b * X + X > NC - MP && b * X < NC;
        // model position of local position 0 (inside the model also where this CTA owns nothing)
        const int base = min(u0 + c0, a.nx - 1);
        const uint16_t *idx_j = a.idx + (long long)j * a.idx_jstride;
        float4 *ckpt = a.ckpt_mode != 0
                           ? reinterpret_cast<float4 *>(a.ckpt_items) + ((long long)it * csize + crank) * a.nslab * pe
                           : work;

        for (int i = threadIdx.x; i < (NEXT + 4 * MP) * ROW; i += blockDim.x) smem[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncthreads();
        if (a.ckpt_mode != 2) {
            for (int k = grp.seg_begin; k < grp.seg_begin + grp.nseg; ++k) {
                const int4 sg = a.segs[k];
                const int r0 = sg.z - u0;
                const int lo = max(r0, c0 - MP), hi = min(r0 + sg.w, c0 + NC + MP);
                const cpx *ws = a.wave + a.shot_off[sg.x] + (long long)j * sg.w;
                const int sq = sg.y & 3, sh = (sg.y >> 2) & 1, sv = sg.y >> 3;  // lane, half of the pair, vector
                for (int x = lo + (int)threadIdx.x; x < hi; x += blockDim.x) {
                    const cpx v = ws[x - r0];
                    const int pos = x - c0 + MP;
                    float *f = reinterpret_cast<float *>(ext + (size_t)pos * ROW + wide_col<Q>(pos, sq, sv));
                    f[sh] = v.re;
                    f[2 + sh] = v.im;
                }
            }
        }
        cluster_arrive();
        cluster_wait();

        if (warp_active) {
            // aperture masks of this lane's four slots: bit 8 v + jj, output jj of slot q + 4 v
            unsigned in = 0;
            {
                const bool blk_active = b * X < own;
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const int slot = q + 4 * v;
                    const int16_t *orow = (blk_active && slot < grp.nslots)
                                              ? a.owner + grp.owner_off + (long long)slot * grp.owner_stride + c0 + b * X
                                              : nullptr;
                    int16_t o[X];
                    load_owner<X>(orow, o);
#pragma unroll
                    for (int jj = 0; jj < X; ++jj) in |= (o[jj] >= 0 && b * X + jj < own ? 1u : 0u) << (8 * v + jj);
                }
            }
            const int iw0 = base + warp * (P * X) - MP; // model position of the warp's first row number
            uint16_t *cur = idxw, *nxt = idxw + NI;
            auto load_idx = [&](uint16_t *dst, int l) {
                const uint16_t *row = idx_j + (long long)l * a.idx_lstride;
                for (int i = lane; i < NI; i += 32) dst[i] = row[min(max(iw0 + i, 0), a.nx - 1)];
            };
            load_idx(cur, a.ckpt_mode == 2 ? (a.nslab - 1) * D : 0);
            __syncwarp();
            unsigned op = 0;  // operations of this item
            int next_l = -1;  // depth step whose row numbers the current operation fetches
            const long long prow = (long long)(b * X) * ROW + q;  // this lane's A of its block, in a plane

            // rows of the operation: neighbours' rows of the last one, or the halo from the next CTA
            auto begin = [&](int nl) {
                if (op > 0) {
                    wait(s_wr + warp, n_op - 1, false);
                    if (hb_left || hb_right) {
                        const unsigned ex = hb_base + op - 1;
                        const float4 *hs = stg + (size_t)(op & 1) * 2 * MP * ROW;
                        if (hb_left) {
                            wait(s_hb + (ex & 1), ex >> 1, true);
                            for (int i = lane; i < MP * ROW; i += 32) ext[i] = hs[i];
                        }
                        if (hb_right) {
                            wait(s_hb + 2 + (ex & 1), ex >> 1, true);
                            for (int i = lane; i < MP * ROW; i += 32) ext[(NC + MP) * ROW + i] = hs[MP * ROW + i];
                        }
                        __syncwarp();
                    }
                }
                next_l = nl;
                if (nl >= 0 && lane < (NI + 63) / 64 + 1)
                    asm volatile("prefetch.global.L1 [%0];" ::"l"(idx_j + (long long)nl * a.idx_lstride +
                                                                 min(max(iw0 + lane * 64, 0), a.nx - 1)));
            };
            auto signal = [&](unsigned long long *bars) {
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(bars + wl);
                    mbar_arrive(bars + wr);
                }
            };
            // end of an operation: its result into this warp's rows (and the neighbouring CTA's staging)
            auto commit = [&](float (&acc)[X][8]) {
                signal(s_rd);
                const int par = (op + 1) & 1;
                if (push_left) {
                    float4 *dst = stg + (size_t)(par * 2 + 1) * MP * ROW;
#pragma unroll
                    for (int jj = 0; jj < X; ++jj) {
                        const int x = b * X + jj;
                        if (x < MP) {
                            const int pr = NC + MP + x;
                            const unsigned ra = map_rank(dst + (size_t)x * ROW, crank - 1);
                            st_cluster(ra + wide_col<Q>(pr, q, 0) * 16, make_float4(acc[jj][0], acc[jj][1], acc[jj][2], acc[jj][3]));
                            st_cluster(ra + wide_col<Q>(pr, q, 1) * 16, make_float4(acc[jj][4], acc[jj][5], acc[jj][6], acc[jj][7]));
                        }
                    }
                }
                if (push_right) {
                    float4 *dst = stg + (size_t)(par * 2) * MP * ROW;
#pragma unroll
                    for (int jj = 0; jj < X; ++jj) {
                        const int x = b * X + jj - (NC - MP);
                        if (x >= 0) {
                            const unsigned ra = map_rank(dst + (size_t)x * ROW, crank + 1);
                            st_cluster(ra + wide_col<Q>(x, q, 0) * 16, make_float4(acc[jj][0], acc[jj][1], acc[jj][2], acc[jj][3]));
                            st_cluster(ra + wide_col<Q>(x, q, 1) * 16, make_float4(acc[jj][4], acc[jj][5], acc[jj][6], acc[jj][7]));
                        }
                    }
                }
                if (hb_left || hb_right) {
                    __syncwarp();
                    if (lane == 0) {
                        const unsigned ex = hb_base + op;
                        if (hb_left) mbar_arrive_cluster(map_rank(s_hb + 2 + (ex & 1), crank - 1));
                        if (hb_right) mbar_arrive_cluster(map_rank(s_hb + (ex & 1), crank + 1));
                    }
                }
                wait(s_rd + warp, n_op, false);
#pragma unroll
                for (int jj = 0; jj < X; ++jj) {
                    const int pr = b * X + MP + jj;
                    float4 *dst = ext + (size_t)pr * ROW;
                    dst[wide_col<Q>(pr, q, 0)] = make_float4(acc[jj][0], acc[jj][1], acc[jj][2], acc[jj][3]);
                    dst[wide_col<Q>(pr, q, 1)] = make_float4(acc[jj][4], acc[jj][5], acc[jj][6], acc[jj][7]);
                }
                signal(s_wr);
                ++op;
                ++n_op;
            };
            // row numbers of the next step: into shared memory after the current ones have been used
            auto next_idx = [&]() {
                if (next_l < 0) return;
                load_idx(nxt, next_l);
                uint16_t *t = cur; cur = nxt; nxt = t;
                __syncwarp();
            };
            auto mask = [&](float (&acc)[X][8]) {
                if (in == 0xffffffffu) return;
#pragma unroll
                for (int jj = 0; jj < X; ++jj) {
#pragma unroll
                    for (int v = 0; v < 4; ++v)
                        if (!((in >> (8 * v + jj)) & 1u)) acc[jj][4 * (v >> 1) + (v & 1)] = acc[jj][4 * (v >> 1) + 2 + (v & 1)] = 0.f;
                }
            };
            auto load_in = [&](int row, float4 &va, float4 &vb) {
                const float4 *r = ext + (size_t)row * ROW + 2 * q;
                const int sw = (row >> 3) & 1;
                va = r[sw];
                vb = r[sw ^ 1];
            };
            auto zero = [&](float (&acc)[X][8]) {
#pragma unroll
                for (int jj = 0; jj < X; ++jj)
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[jj][e] = 0.f;
            };
            auto load_plane = [&](float (&acc)[X][8], const float4 *plane) {
#pragma unroll
                for (int jj = 0; jj < X; ++jj) {
                    const float4 va = plane[prow + jj * ROW], vb = plane[prow + jj * ROW + Q];
                    acc[jj][0] = va.x; acc[jj][1] = va.y; acc[jj][2] = va.z; acc[jj][3] = va.w;
                    acc[jj][4] = vb.x; acc[jj][5] = vb.y; acc[jj][6] = vb.z; acc[jj][7] = vb.w;
                }
            };
            auto store_plane = [&](const float (&acc)[X][8], float4 *plane) {
#pragma unroll
                for (int jj = 0; jj < X; ++jj) {
                    plane[prow + jj * ROW] = make_float4(acc[jj][0], acc[jj][1], acc[jj][2], acc[jj][3]);
                    plane[prow + jj * ROW + Q] = make_float4(acc[jj][4], acc[jj][5], acc[jj][6], acc[jj][7]);
                }
            };
            const int srow0 = b * X + MP - M;
            const int iw = p * X + MP;  // row number of the block's first output in cur[]
            const int nmid = (L - X + 1) / 2;

            // the ring, as in migrate_wide_kernel
            unsigned rcopy[4];
            const int rh = q & 1;
            auto ring_pair = [&](int v, bool both) {
                if (!both && rh) return;
                const int sl = (v + rh) & (kRingSlots - 1);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int o = (q >> 1) + 2 * i;
                    const int pr = v + rh + ((X - o) >> 1);
                    const bool ok = (unsigned)pr < (unsigned)npairs;
                    cp_async16_zfill(ringb + o * kRingSlots + sl, tabb + rcopy[i] + (ok ? pr : 0) * 16, ok ? 16u : 0u);
                }
            };
            // forward step: acc = A_l S of this block, rows of the outputs
            auto fir_forward_w = [&](float (&acc)[X][8]) {
                zero(acc);
                const char *row[X];
                if (RING) {
                    // (copied at the end of the operation before: no faster)
#pragma unroll
                    for (int i = 0; i < 4; ++i) rcopy[i] = (unsigned)cur[iw + (q >> 1) + 2 * i] * (unsigned)row_bytes;
                    ring_pair(-4, true);
                    ring_pair(-2, true);
                    cp_async_commit();
                    cp_async_wait<0>();
                    __syncwarp();
                } else {
#pragma unroll
                    for (int jj = 0; jj < X; ++jj) row[jj] = tabb + (size_t)cur[iw + jj] * row_bytes;
                }
                // pair pr of output jj, from ring iteration u
                auto pair = [&](int jj, int u) {
                    return RING ? ringb[jj * kRingSlots + (u & (kRingSlots - 1))]
                                : __ldg(reinterpret_cast<const float4 *>(row[jj]) + u + ((X - jj) >> 1));
                };
                float4 tp[X];
#pragma unroll
                for (int t = 0; t < X - 1; ++t) {
                    float4 va, vb;
                    load_in(srow0 + t, va, vb);
#pragma unroll
                    for (int jj = 0; jj < X; ++jj) {
                        const int k = t - jj;
                        if (k >= 0) {
                            if ((k & 1) == 0) tp[jj] = pair(jj, (k >> 1) - ((X - jj) >> 1));
                            wide_mac<1>(acc[jj], (k & 1) ? tp[jj].z : tp[jj].x, (k & 1) ? tp[jj].w : tp[jj].y, va, vb);
                        }
                    }
                    if (RING && t == 2) {
                        ring_pair(0, true);
                        cp_async_commit();
                    }
                }
                int rowi = srow0 + X - 1;
                for (int u = 0; u < nmid; ++u, rowi += 2) {
                    if (RING && !(u & 1)) {
                        ring_pair(u + 2, true);
                        cp_async_commit();
                        cp_async_wait<1>();
                        __syncwarp();
                    }
                    {
                        float4 va, vb;
                        load_in(rowi, va, vb);
#pragma unroll
                        for (int jj = 0; jj < X; ++jj) {
                            if (jj & 1) tp[jj] = pair(jj, u);
                            wide_mac<1>(acc[jj], (jj & 1) ? tp[jj].x : tp[jj].z, (jj & 1) ? tp[jj].y : tp[jj].w, va, vb);
                        }
                    }
                    {
                        float4 va, vb;
                        load_in(rowi + 1, va, vb);
#pragma unroll
                        for (int jj = 0; jj < X; ++jj) {
                            if (!(jj & 1)) tp[jj] = pair(jj, u);
                            wide_mac<1>(acc[jj], (jj & 1) ? tp[jj].z : tp[jj].x, (jj & 1) ? tp[jj].w : tp[jj].y, va, vb);
                        }
                    }
                }
                if (RING) {
                    ring_pair((nmid + 3) & ~1, !(nmid & 1));
                    cp_async_commit();
                }
#pragma unroll
                for (int e = 0; e < X - 1; ++e) {
                    float4 va, vb;
                    load_in(srow0 + L + e, va, vb);
                    if (RING && (e & 1) == 0 && !((nmid + (e >> 1)) & 1)) {
                        if (e < 4) cp_async_wait<1>();
                        else cp_async_wait<0>();
                        __syncwarp();
                    }
#pragma unroll
                    for (int jj = 0; jj < X; ++jj) {
                        if (jj > e) {
                            const bool even = ((1 + e - jj) & 1) == 0;
                            if (even) tp[jj] = pair(jj, nmid + (e >> 1));
                            wide_mac<1>(acc[jj], even ? tp[jj].x : tp[jj].z, even ? tp[jj].y : tp[jj].w, va, vb);
                        }
                    }
                }
            };
            // transposed step: output jj takes tap jj + 2M - t of the row of input t
            auto fir_transposed_w = [&](float (&acc)[X][8]) {
                zero(acc);
                auto row_of = [&](int t) {
                    return reinterpret_cast<const float4 *>(tabb + (size_t)cur[iw - M + t] * row_bytes);
                };
                // taps k0 .. of one input for outputs j0 .. j1 - 1 (compile-time), k0 even or odd
                auto run = [&](const float4 *rp, bool odd, int j0, int j1, const float4 &va, const float4 &vb) {
                    float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int jj = 0; jj < X; ++jj) {
                        if (jj >= j0 && jj < j1) {
                            const int i = jj - j0 + (odd ? 1 : 0);  // tap of the run, from its first pair
                            if ((i & 1) == 0 || jj == j0) c = __ldg(rp + (i >> 1));
                            wide_mac<1>(acc[jj], (i & 1) ? c.z : c.x, (i & 1) ? c.w : c.y, va, vb);
                        }
                    }
                };
                // t = 0 .. X - 2: outputs 0 .. t, taps 2M - t .. 2M
#pragma unroll
                for (int t = 0; t < X - 1; ++t) {
                    float4 va, vb;
                    load_in(srow0 + t, va, vb);
                    run(row_of(t) + (M - ((t + 1) >> 1)), (t & 1) != 0, 0, t + 1, va, vb);
                }
                // all outputs: t odd, then t + 1
                for (int t = X - 1; t < L - 1; t += 2) {
                    {
                        float4 va, vb;
                        load_in(srow0 + t, va, vb);
                        run(row_of(t) + (M - ((t + 1) >> 1)), true, 0, X, va, vb);
                    }
                    {
                        float4 va, vb;
                        load_in(srow0 + t + 1, va, vb);
                        run(row_of(t + 1) + (M - ((t + 1) >> 1)), false, 0, X, va, vb);
                    }
                }
                // t = L + e: outputs e + 1 .., taps 0 ..
#pragma unroll
                for (int e = 0; e < X - 1; ++e) {
                    float4 va, vb;
                    load_in(srow0 + L + e, va, vb);
                    run(row_of(L + e), false, e + 1, X, va, vb);
                }
            };

            // Phase 1: checkpoints S_{cD} (skipped when they come from the cache)
            if (a.ckpt_mode != 2) {
                float acc[X][8];
#pragma unroll
                for (int jj = 0; jj < X; ++jj) {
                    float4 va, vb;
                    load_in(b * X + MP + jj, va, vb);
                    acc[jj][0] = va.x; acc[jj][1] = va.y; acc[jj][2] = va.z; acc[jj][3] = va.w;
                    acc[jj][4] = vb.x; acc[jj][5] = vb.y; acc[jj][6] = vb.z; acc[jj][7] = vb.w;
                }
                store_plane(acc, ckpt);
                for (int l = 0; l < (a.nslab - 1) * D; ++l) {
                    begin(l + 1);
                    fir_forward_w(acc);
                    mask(acc);
                    if ((l + 1) % D == 0) store_plane(acc, ckpt + (long long)((l + 1) / D) * pe);
                    next_idx();
                    commit(acc);
                }
            }
            // Phase 2: slabs in reverse depth order
            for (int c = a.nslab - 1; c >= 0; --c) {
                const int lb = c * D, le = min(lb + D, a.nextrap);
                float acc[X][8];
                // steps of the slab that apply A: not the last one above the deepest slab
                const int lf = c == a.nslab - 1 ? le : le - 1;
                if (c != a.nslab - 1 || a.ckpt_mode == 2) {
                    begin(-1);
                    load_plane(acc, ckpt + (long long)c * pe);
                    commit(acc);
                }
                for (int l = lb; l < le; ++l) {
                    // the row numbers of the last step serve the first transposed one too
                    begin(l + 1 < le ? l + 1 : -1);
                    if (l >= lf) {
                        // S_le is the next checkpoint and not needed here; V_{le-1} is what the slab below left
                        load_plane(acc, save);
                    } else {
                        fir_forward_w(acc);
                        mask(acc);
                        if (l + 1 < le) {
                            store_plane(acc, slabbuf + (long long)(l - lb) * pe);
                        } else {
                            // V_{nextrap-1} = m S_nextrap
                            const float *mrow = a.refl + (long long)(le - 1) * a.nx + base;
#pragma unroll
                            for (int jj = 0; jj < X; ++jj) {
                                const float m = b * X + jj < own ? mrow[b * X + jj] : 0.f;
#pragma unroll
                                for (int e = 0; e < 8; ++e) acc[jj][e] *= m;
                            }
                        }
                        next_idx();
                    }
                    commit(acc);
                }
                for (int l = le - 1; l >= lb; --l) {
                    begin(l > lb ? l - 1 : (c > 0 ? (c - 1) * D : -1));
                    const float4 *Sl = (l > lb) ? slabbuf + (long long)(l - 1 - lb) * pe : ckpt + (long long)c * pe;
                    const float *mrow = a.refl + (long long)(l - 1) * a.nx + base;
                    if (l > 0) {
                        // the source plane the emission after the taps reads, into L1
#pragma unroll
                        for (int jj = 0; jj < X; jj += Q)
                            asm volatile("prefetch.global.L1 [%0];" ::"l"(Sl + (long long)(b * X + jj + q) * ROW));
                    }
                    fir_transposed_w(acc);
                    mask(acc);
                    if (l > 0) {
#pragma unroll
                        for (int jj = 0; jj < X; ++jj) {
                            const float m = b * X + jj < own ? mrow[b * X + jj] : 0.f;
                            const float4 sa = Sl[prow + jj * ROW], sb = Sl[prow + jj * ROW + Q];  // zero outside the apertures
                            const float s[8] = {sa.x, sa.y, sa.z, sa.w, sb.x, sb.y, sb.z, sb.w};
                            if (b * X + jj < own) {
#pragma unroll
                                for (int e = 0; e < 8; ++e) acc[jj][e] = fmaf(m, s[e], acc[jj][e]);
                            }
                        }
                    }
                    if (l == lb && l > 0) store_plane(acc, save);
                    next_idx();
                    commit(acc);
                }
            }
            hb_base += op;
        } else {
            // edge barriers advance for all warps alike (an inactive warp may be an edge in a later item)
            const int steps = (a.ckpt_mode != 2 ? (a.nslab - 1) * D : 0) + 2 * a.nextrap + a.nslab - (a.ckpt_mode == 2 ? 0 : 1);
            hb_base += steps;
        }
        __syncthreads();
        // ext holds U_0 = F* m for this CTA's positions
        for (int k = grp.seg_begin; k < grp.seg_begin + grp.nseg; ++k) {
            const int4 sg = a.segs[k];
            const int r0 = sg.z - u0;
            const int lo = max(r0, c0), hi = min(r0 + sg.w, c0 + own);
            cpx *ds = a.data + a.shot_off[sg.x] + (long long)j * sg.w;
            const int sq = sg.y & 3, sh = (sg.y >> 2) & 1, sv = sg.y >> 3;
            for (int x = lo + (int)threadIdx.x; x < hi; x += blockDim.x) {
                const int pos = x - c0 + MP;
                const float *f = reinterpret_cast<const float *>(ext + (size_t)pos * ROW + wide_col<Q>(pos, sq, sv));
                ds[x - r0] = cpx{f[sh], f[2 + sh]};
            }
        }
        __syncthreads();
    }
    cluster_arrive();
    cluster_wait();
}

}  // namespace img2d
