// Row-split migration kernel: surveys of few shots, forward/backward table pairs.
//
// With one or two lane slots an operator row feeds 8 L G FMAs (G slots) and is used once, so what
// bounds the kernel is how fast rows of 8 L bytes reach the registers, not the FMA pipe.  A lane per
// output (the earlier single-CTA kernels) makes every 16-byte load of a warp touch 32 cache lines,
// one L1 tag lookup each.  Here four lanes (a quad) share a block of X outputs and split the *taps*:
// lane r holds taps [r Q, r Q + Q), Q = 2 NP, of all X rows, so a quad reads 128 consecutive bytes of
// one row with one 32-byte load per lane, and the partial sums are combined by a reduce-scatter over
// the quad (two exchanges) once per block.  The table is laid out for that order
// (rows_table_kernel).  Rows come through L1: consecutive depth steps of one frequency read nearly
// the same rows (k = w/v changes slowly with depth), and L1 keeps what shared memory leaves free.
//
// Measured on a B200 (whole call, against the single-CTA kernels before): one shot of 1024 x 500 with
// 256 frequencies and 31 taps 10.7 -> 3.8 ms (17 TFLOP/s), 4 shots of 320 x 200, 64 frequencies,
// 25 taps 0.97 -> 0.45 ms, 9 shots of 151 x 136, 60 frequencies, 43 taps and two tables 3.50 -> 0.63 ms.
// In the one-shot case L1 serves 68% of the row sectors and its data pipe is 54% busy, issue slots 51%;
// with 12 to 16 warps of 128 registers per SM neither fills up.
//
// Wavefields of an item (G slots x one frequency) stay in shared memory, two buffers in turn, one
// barrier per depth step.  A position is one float4 (S.re, S.im, R.re, R.im) with one slot, and with
// two slots a, b one float4 of S (a.re, b.re, a.im, b.im) and one of R, so that the multiply-adds are
// packed (FFMA2); R is conjugated in the single-table mode.  One unused float4 after every 8 positions
// spreads a quad's four tap ranges over the banks.  The operator row offsets come from shared memory,
// where each step stores those of the step after next.
//
// Image: the first item of a CTA stores its rows of the CTA's partial image (nothing has to be zeroed
// or read), later ones add with Kahan compensation; the reduction reads what the CTA's item count
// says was written.
#pragma once
#include "wlsq_kernels.cuh"

namespace img2d {

constexpr int kRowsThreads = 512;        // most threads per CTA
constexpr int kRowsX = 4;                // outputs per quad
constexpr int kRowsWarpPos = 8 * kRowsX; // positions of one warp's pass

__host__ __device__ inline int rows_np(int L)
{
    const int np = (L + 7) / 8;
    return np == 9 ? 10 : np;
}

// floats of one table row: 4 lanes x 2 NP taps x (re, im), forward and backward in turn for two tables
__host__ __device__ inline int rows_row_floats(int L, bool two) { return 16 * rows_np(L) * (two ? 2 : 1); }

__host__ __device__ constexpr int rows_pad(int x) { return x + (x >> 3); }

// Lane r of a quad holds taps [s_r, s_r + Q), Q = 2 NP; every tap has a lane.  s_0 = 0 and s_3 = L - Q,
// or one more, where the last tap of lane 3 does not exist and is skipped.  The two quads of a quarter
// warp work on blocks `apart` blocks apart.  The freedom in s_1, s_2, s_3 and `apart` is spent on the
// quarter warp's shared-memory reads (16 bytes a lane): the choice with the fewest bank conflicts
// (1.0 to 2.0 passes a read; 31 taps in ranges of 8, one tap missing: 1.0 against 2.0 without it,
// 3.42 against 3.68 ms for one shot of 1024 x 500, 256 frequencies).
struct RowsStarts {
    int s[4];
    int apart;      // 1, 2 or 4
    double passes;  // of a quarter warp's read
};
inline RowsStarts rows_starts(int L)
{
    const int X = kRowsX, Q = 2 * rows_np(L);
    RowsStarts best{{0, 0, 0, 0}, 1, 1.0};
    int best_cost = 1 << 30;
    for (int apart = 1; apart <= 4; apart *= 2)
        for (int s3 = L - Q; s3 <= L - Q + 1 && s3 <= 3 * Q; ++s3)
            for (int s1 = 0; s1 <= Q && s1 <= s3; ++s1)
                for (int s2 = s1; s2 <= s1 + Q && s2 <= s3; ++s2) {
                    if (s3 - s2 > Q) continue;
                    const int s[4] = {0, s1, s2, s3};
                    const int extra = (s3 > L - Q ? 3 : 0) + (apart > 1 ? 1 : 0);
                    int cost = extra;
                    for (int x = 0; x < 64; ++x) {
                        int at[8], banks[8] = {}, worst = 0;
                        for (int i = 0; i < 8; ++i) {
                            at[i] = rows_pad(x + (i >> 2) * apart * X + s[i & 3]);
                            bool same = false;  // the same address is read once
                            for (int k = 0; k < i; ++k) same |= at[k] == at[i];
                            if (!same) worst = worst > ++banks[at[i] & 7] ? worst : banks[at[i] & 7];
                        }
                        cost += worst;
                    }
                    if (cost < best_cost) {
                        best_cost = cost;
                        best = RowsStarts{{s[0], s[1], s[2], s[3]}, apart, (cost - extra) / 64.0};
                    }
                }
    return best;
}

// Float4 entries of one slot's buffer for a window of W positions: M (rounded up to 8) zeros on
// either side, W rounded up to whole warps.
__host__ __device__ inline int rows_positions(int W, int L)
{
    const int M = (L - 1) / 2;
    const int left = (M + 7) / 8 * 8;
    const int wp = (W + kRowsWarpPos - 1) / kRowsWarpPos * kRowsWarpPos;
    return left + wp + left;
}
__host__ __device__ inline size_t rows_smem_bytes(int G, int W, int L)
{
    const int np = rows_positions(W, L), wp = (W + kRowsWarpPos - 1) / kRowsWarpPos * kRowsWarpPos;
    return 2 * (size_t)G * (rows_pad(np) + 1) * 16 + 3 * (size_t)wp * 4 + (size_t)G * (wp / kRowsX);
}

// Padded copy of the compact table in the kernel's order.  Row: chunks of 4 lanes x 32 bytes (4 taps
// each), then for odd NP one chunk of 4 lanes x 16 bytes (2 taps); lane r's chunk c holds taps
// s_r + 4 c ...; each chunk of the backward table follows the forward one.  Where the ranges of two,
// three or four lanes overlap, each holds a half, a quarter (the first of three a half) or a quarter
// of the tap: the products then add up to the tap's (scaling by a power of two is exact) and
// infinities and NaN come out as from the whole tap.
__global__ void rows_table_kernel(const cpx *__restrict__ tabF, const cpx *__restrict__ tabB, int stride, int L,
                                  int NP, RowsStarts st, int nk, float *__restrict__ out)
{
    const int nt = tabB ? 2 : 1;
    const int per_row = 8 * NP * nt;  // complex elements
    const long long total = (long long)nk * per_row;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int row = (int)(e / per_row), i = (int)(e % per_row);
        const int c = i / (16 * nt), ic = i % (16 * nt);          // chunk, element inside it
        const int lane_taps = c < NP / 2 ? 4 : 2;                 // the odd half chunk is last
        const int which = ic / (4 * lane_taps), il = ic % (4 * lane_taps);
        const int r = il / lane_taps, k = st.s[r] + 4 * c + il % lane_taps;
        int m = 0, before = 0;  // lanes that hold tap k, and those of them below r
        for (int q = 0; q < 4; ++q) {
            const int d = k - st.s[q];
            if (d >= 0 && d < 2 * NP) {
                ++m;
                before += q < r ? 1 : 0;
            }
        }
        const float w = m == 1 ? 1.f : (m == 2 || (m == 3 && before == 0) ? 0.5f : 0.25f);
        const cpx v = k < L ? (which ? tabB : tabF)[(long long)row * stride + k] : cpx{0.f, 0.f};
        out[2 * e] = w * v.re;
        out[2 * e + 1] = w * v.im;
    }
}

struct RowTaps {
    float f[8];  // 4 taps (re, im)
};

__device__ __forceinline__ void rows_load8(RowTaps &t, const char *p)
{
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(t.f[0]), "=f"(t.f[1]), "=f"(t.f[2]), "=f"(t.f[3]), "=f"(t.f[4]), "=f"(t.f[5]), "=f"(t.f[6]), "=f"(t.f[7])
        : "l"(p));
}

// G: lane slots per item.  NP: tap pairs per lane.  TWO: forward and backward table; else the receiver
// uses the conjugated forward rows.
template <int G, int NP, bool TWO>
__global__ void __launch_bounds__(kRowsThreads, 1) migrate_rows_kernel(MigrateArgs a)
{
    constexpr int X = kRowsX, Q = 2 * NP;
    constexpr int NT = TWO ? 2 : 1;
    constexpr int ROWB = 64 * NP * NT;   // bytes of one table row
    constexpr int WP_POS = kRowsWarpPos;
    constexpr int NF = (Q + 3) / 4;      // chunks of up to 4 taps
    constexpr int R = X / 4;             // outputs a lane keeps after the reduce-scatter
    const int M = a.M, L = 2 * M + 1;
    const int left = (M + 7) / 8 * 8;
    extern __shared__ float4 smem[];
    __shared__ int s_item;
    const int T = blockDim.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = T >> 5;
    const int r = lane & 3, qd = lane >> 3;
    // this quad's place in the warp: the second quad of a quarter warp row_apart blocks on
    const int p = (qd & (a.row_apart - 1)) + ((lane >> 2) & 1) * a.row_apart + (qd & -a.row_apart) * 2;
    const char *tab = reinterpret_cast<const char *>(a.tab_rows);
    const long long plane = (long long)a.nextrap * a.nx;
    float *part = a.partial ? a.partial + (long long)blockIdx.x * plane : nullptr;
    float *comp = a.comp ? a.comp + (long long)blockIdx.x * plane : nullptr;
    const int tap0 = a.row_start[r];  // this lane's first tap
    const bool last_tap = tap0 + Q <= L;
    // first input of window position 0: entry e8 of 8-row hi8 (block starts are multiples of 8 X plus p X)
    const int first_in = left - M + tap0 + (p * X & 7);
    const int hi8 = first_in >> 3, e8 = first_in & 7;
    int done = a.visits ? a.visits[blockIdx.x] : 0;  // items this CTA's partial image holds
    bool first = true;

    // chunk c of one row (at byte offset off): this lane's taps
    struct Taps {
        RowTaps t[NT];
    };
    auto load_taps = [&](Taps &o, unsigned off, int c) {
        if (Q - 4 * c >= 4) {
            const char *h = tab + (size_t)(off + r * 32) + c * 128 * NT;
            rows_load8(o.t[0], h);
            if (TWO) rows_load8(o.t[NT - 1], h + 128);
        } else {
            // half chunk: 2 taps, 16 bytes per lane
            const char *h = tab + (size_t)(off + r * 16) + c * 128 * NT;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const float4 v = __ldg(reinterpret_cast<const float4 *>(h + n * 64));
                o.t[n].f[0] = v.x; o.t[n].f[1] = v.y; o.t[n].f[2] = v.z; o.t[n].f[3] = v.w;
            }
        }
    };
    auto load_off = [&](unsigned (&o)[X], const unsigned *src) {
#pragma unroll
        for (int i = 0; i < X; i += 4) {
            const uint4 v = *reinterpret_cast<const uint4 *>(src + i);
            o[i] = v.x; o[i + 1] = v.y; o[i + 2] = v.z; o[i + 3] = v.w;
        }
    };

    for (;;) {
        int it;
        if (a.n_items <= (int)gridDim.x) {
            // every CTA has at most one item: no queue, and no second visit of its partial image
            it = first ? (int)blockIdx.x : a.n_items;
        } else {
            if (threadIdx.x == 0) s_item = atomicAdd(a.counter, 1);
            __syncthreads();
            it = s_item;
        }
        __syncthreads();
        if (it >= a.n_items) break;
        first = false;
        const int2 item = a.items[it];
        const GroupDesc grp = a.groups[item.x];
        const int j = item.y, u0 = grp.u0, W = grp.W;
        const int nwb = (W + WP_POS - 1) / WP_POS, wp = nwb * WP_POS;
        const int npos = left + wp + left;
        const int ns = rows_pad(npos) + 1;  // entries of one slot's buffer
        float4 *bufA = smem, *bufB = smem + (size_t)G * ns;
        // row offsets of this step, the next and the one after
        unsigned *off0 = reinterpret_cast<unsigned *>(smem + (size_t)2 * G * ns), *off1 = off0 + wp, *off2 = off1 + wp;
        unsigned char *mask = reinterpret_cast<unsigned char *>(off2 + wp);  // [G][wp / X]
        for (int i = threadIdx.x; i < 2 * G * ns; i += T) smem[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        const uint16_t *idx_j = a.idx + (long long)j * a.idx_jstride;
        for (int x = threadIdx.x; x < wp; x += T) {
            const int xm = min(u0 + x, a.nx - 1);
            off0[x] = (unsigned)idx_j[xm] * (unsigned)ROWB;
            off1[x] = a.nextrap > 1 ? (unsigned)idx_j[a.idx_lstride + xm] * (unsigned)ROWB : 0u;
            off2[x] = 0u;  // with two steps the last one looks ahead to it
        }
        for (int i = threadIdx.x; i < G * (wp / X); i += T) {
            const int g = i / (wp / X), b = i % (wp / X);
            unsigned m = 0;
            if (g < grp.nslots) {
                const int16_t *orow = a.owner + grp.owner_off + (long long)g * grp.owner_stride;
                for (int jj = 0; jj < X; ++jj) m |= (b * X + jj < W && orow[b * X + jj] >= 0 ? 1u : 0u) << jj;
            }
            mask[i] = (unsigned char)m;
        }
        __syncthreads();
        for (int k = grp.seg_begin; k < grp.seg_begin + grp.nseg; ++k) {
            const int4 sg = a.segs[k];
            const cpx *ws = a.wave + a.shot_off[sg.x] + (long long)j * sg.w;
            const cpx *rs = a.shot + a.shot_off[sg.x] + (long long)j * sg.w;
            for (int i = threadIdx.x; i < sg.w; i += T) {
                const cpx S = ws[i], V = rs[i];
                const int at = rows_pad(left + sg.z - u0 + i);
                if (G == 2) {
                    float *fs = reinterpret_cast<float *>(bufA + at) + sg.y, *fr = reinterpret_cast<float *>(bufA + ns + at) + sg.y;
                    fs[0] = S.re;
                    fs[2] = S.im;
                    fr[0] = V.re;
                    fr[2] = TWO ? V.im : -V.im;
                } else {
                    bufA[at] = make_float4(S.re, S.im, V.re, TWO ? V.im : -V.im);
                }
            }
        }
        // The taps of a row's first chunk are always loaded one block ahead (across the step boundary
        // too), those of a later chunk as the chunk before is used up: the registers of a row's taps
        // are refilled as soon as they have been read.
        unsigned off[X];
        Taps tp[X];
        if (warp < nwb) {
            load_off(off, off0 + (warp * 8 + p) * X);
#pragma unroll
            for (int jj = 0; jj < X; ++jj) load_taps(tp[jj], off[jj], 0);
        }
        __syncthreads();

        for (int l = 0; l < a.nextrap; ++l) {
            const bool more = l + 2 < a.nextrap;
            const uint16_t *inext = idx_j + (long long)(l + 2) * a.idx_lstride;
            float *prow = part ? part + (long long)l * a.nx : nullptr;
            float *crow = comp ? comp + (long long)l * a.nx : nullptr;
            if (prow && done == 0) {
                // first visit: positions outside this item's window start at zero
                for (int x = threadIdx.x; x < u0; x += T) prow[x] = 0.f;
                for (int x = u0 + W + threadIdx.x; x < a.nx; x += T) prow[x] = 0.f;
            }
            for (int wb = warp; wb < nwb; wb += nwarps) {
                const int b = wb * 8 + p;       // this quad's block
                const int xb = b * X;           // its first output, window position
                // operator rows of the outputs this lane keeps, two steps ahead: loaded now, stored at
                // the end of the block
                unsigned nidx[R];
                if (more) {
#pragma unroll
                    for (int i = 0; i < R; ++i) nidx[i] = inext[min(u0 + xb + r * R + i, a.nx - 1)];
                }
                // Kahan values of the outputs this lane keeps
                float ps[R], pc[R];
                if (prow && done > 0) {
#pragma unroll
                    for (int i = 0; i < R; ++i) {
                        const int x = xb + r * R + i;
                        ps[i] = x < W ? prow[u0 + x] : 0.f;
                        pc[i] = x < W && done > 1 ? crow[u0 + x] : 0.f;
                    }
                }
                float acc[X][G][4];
                // inputs i = 0 ... Q + X - 2 of this lane, from position left + xb - M + tap0: that is
                // 8-row hi, element e + i, one pad entry further after each row end
                const float4 *src = bufA + (hi8 + (xb >> 3)) * 9 + e8;
                float4 win[X + 3][G];
                auto load_in = [&](int i, float4 (&v)[G]) {
                    const float4 *q = src + ((i & 7) >= 8 - e8 ? (i >> 3) + 1 : (i >> 3));
#pragma unroll
                    for (int g = 0; g < G; ++g) v[g] = q[(size_t)g * ns + i];
                };
#pragma unroll
                for (int i = 0; i < X - 1; ++i) load_in(i, win[i]);
#pragma unroll
                for (int c = 0; c < NF; ++c) {
                    const int nt = Q - 4 * c < 4 ? Q - 4 * c : 4;  // taps of this chunk (4, or 2 in the last)
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (i < nt) load_in(4 * c + X - 1 + i, win[X - 1 + i]);
                    if (c == NF - 1) {
                        // row offsets of this warp's next block: of this step, or the first of the next
                        const unsigned *os = wb + nwarps < nwb ? off0 + xb + nwarps * WP_POS
                                                               : off1 + (warp * 8 + p) * X;
                        load_off(off, os);
                    }
                    auto tap = [&](int jj, int d) {
                        const float fr = tp[jj].t[0].f[2 * d], fi = tp[jj].t[0].f[2 * d + 1];
                        const float br = tp[jj].t[NT - 1].f[2 * d], bi = tp[jj].t[NT - 1].f[2 * d + 1];
#pragma unroll
                        for (int g = 0; g < G; ++g) {
                            const float4 v = win[jj + d][g];
                            float (&s)[4] = acc[jj][g];
                            if (G == 2) {
                                // both slots' S (g = 0) or R (g = 1) at once
                                const float tr = g ? br : fr, ti = g ? bi : fi;
                                float2 *s2 = reinterpret_cast<float2 *>(s);
                                const float2 re = make_float2(v.x, v.y), im = make_float2(v.z, v.w);
                                if (c == 0 && d == 0) {
                                    s2[0] = make_float2(tr * v.x, tr * v.y);
                                    s2[1] = make_float2(tr * v.z, tr * v.w);
                                } else {
                                    s2[0] = __ffma2_rn(make_float2(tr, tr), re, s2[0]);
                                    s2[1] = __ffma2_rn(make_float2(tr, tr), im, s2[1]);
                                }
                                s2[0] = __ffma2_rn(make_float2(-ti, -ti), im, s2[0]);
                                s2[1] = __ffma2_rn(make_float2(ti, ti), re, s2[1]);
                                continue;
                            }
                            if (c == 0 && d == 0) {
                                s[0] = fr * v.x; s[1] = fr * v.y; s[2] = br * v.z; s[3] = br * v.w;
                            } else {
                                s[0] = fmaf(fr, v.x, s[0]); s[1] = fmaf(fr, v.y, s[1]);
                                s[2] = fmaf(br, v.z, s[2]); s[3] = fmaf(br, v.w, s[3]);
                            }
                            s[0] = fmaf(-fi, v.y, s[0]); s[1] = fmaf(fi, v.x, s[1]);
                            s[2] = fmaf(-bi, v.w, s[2]); s[3] = fmaf(bi, v.z, s[3]);
                        }
                    };
#pragma unroll
                    for (int jj = 0; jj < X; ++jj) {
#pragma unroll
                        for (int d = 0; d < 4; ++d)
                            if (d < nt && (c < NF - 1 || d < nt - 1)) tap(jj, d);
                        if (c < NF - 1) load_taps(tp[jj], off[jj], c + 1);
                    }
                    if (c == NF - 1) {
                        if (last_tap) {
#pragma unroll
                            for (int jj = 0; jj < X; ++jj) tap(jj, nt - 1);
                        }
#pragma unroll
                        for (int jj = 0; jj < X; ++jj) load_taps(tp[jj], off[jj], 0);
                    }
#pragma unroll
                    for (int i = 0; i < X - 1; ++i)
#pragma unroll
                        for (int g = 0; g < G; ++g) win[i][g] = win[i + 4][g];
                }
                // reduce-scatter over the quad: lane r keeps outputs r R ... r R + R - 1
                const bool hi2 = (r & 2) != 0, hi1 = (r & 1) != 0;
                float img[R];
#pragma unroll
                for (int i = 0; i < R; ++i) img[i] = 0.f;
                static_assert(R == 1, "a lane keeps one of the quad's four outputs");
                float out[G][4];
#pragma unroll
                for (int g = 0; g < G; ++g) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        float h[2];
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const float keep = hi2 ? acc[2 + i][g][e] : acc[i][g][e];
                            const float send = hi2 ? acc[i][g][e] : acc[2 + i][g][e];
                            h[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
                        }
                        const float keep = hi1 ? h[1] : h[0], send = hi1 ? h[0] : h[1];
                        out[g][e] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
                    }
                }
                const int xo = xb + r;  // this lane's output
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    // slot g: its components among out[]
                    float &sr = G == 2 ? out[0][g] : out[g][0], &si = G == 2 ? out[0][2 + g] : out[g][1];
                    float &rr = G == 2 ? out[G - 1][g] : out[g][2], &ri = G == 2 ? out[G - 1][2 + g] : out[g][3];
                    const bool in = (mask[g * (wp / X) + b] >> r) & 1u;
                    if (!in) sr = si = rr = ri = 0.f;
                    const float v = TWO ? sr * rr + si * ri : sr * rr - si * ri;
                    img[0] += v;
                    if (a.image_shots && in) {
                        const int s = a.owner[grp.owner_off + (long long)g * grp.owner_stride + xo];
                        atomicAdd(a.image_shots + (long long)s * a.img_sstride + (long long)l * a.nx + u0 + xo, v);
                    }
                }
#pragma unroll
                for (int g = 0; g < G; ++g)
                    bufB[(size_t)g * ns + rows_pad(left + xo)] = make_float4(out[g][0], out[g][1], out[g][2], out[g][3]);
                if (more) {
#pragma unroll
                    for (int i = 0; i < R; ++i) off2[xb + r * R + i] = nidx[i] * (unsigned)ROWB;
                }
                if (prow) {
#pragma unroll
                    for (int i = 0; i < R; ++i) {
                        const int x = xb + r * R + i;
                        if (x >= W) continue;
                        if (done == 0) {
                            prow[u0 + x] = img[i];
                        } else {
                            const float y = img[i] - pc[i];
                            const float t = ps[i] + y;
                            prow[u0 + x] = t;
                            crow[u0 + x] = (t - ps[i]) - y;
                        }
                    }
                }
            }
            if (prow && done == 1) {
                // the second visit defines the compensation of the whole row
                for (int x = threadIdx.x; x < u0; x += T) crow[x] = 0.f;
                for (int x = u0 + W + threadIdx.x; x < a.nx; x += T) crow[x] = 0.f;
            }
            __syncthreads();
            float4 *t = bufA; bufA = bufB; bufB = t;
            unsigned *o = off0; off0 = off1; off1 = off2; off2 = o;
        }
        if (a.write_back) {
            for (int k = grp.seg_begin; k < grp.seg_begin + grp.nseg; ++k) {
                const int4 sg = a.segs[k];
                cpx *ws = a.wave + a.shot_off[sg.x] + (long long)j * sg.w;
                cpx *rs = a.shot + a.shot_off[sg.x] + (long long)j * sg.w;
                for (int i = threadIdx.x; i < sg.w; i += T) {
                    const int at = rows_pad(left + sg.z - u0 + i);
                    if (G == 2) {
                        const float *fs = reinterpret_cast<const float *>(bufA + at) + sg.y;
                        const float *fr = reinterpret_cast<const float *>(bufA + ns + at) + sg.y;
                        ws[i] = cpx{fs[0], fs[2]};
                        rs[i] = cpx{fr[0], TWO ? fr[2] : -fr[2]};
                    } else {
                        const float4 v = bufA[at];
                        ws[i] = cpx{v.x, v.y};
                        rs[i] = cpx{v.z, TWO ? v.w : -v.w};
                    }
                }
            }
        }
        ++done;
        __syncthreads();
    }
    if (a.visits && threadIdx.x == 0) a.visits[blockIdx.x] = done;
}

}  // namespace img2d
