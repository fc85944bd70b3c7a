// Demigration for few lane slots: the adjoint of wlsq_adjoint.cuh with the row-split kernel's operator
// access (wlsq_rows.cuh: a quad of lanes reads 128 consecutive bytes of an operator row, each lane
// holding its own range of taps).
//
// One item = up to two lane slots x one frequency, one CTA; the complex values of its slots at a
// position form one vector (16 bytes for two slots).  The source is stepped forward once and every
// S_l goes to global memory: into the CTA's work planes, or into the per-item cache that
// IMG2D_SOURCE_KEEP leaves on the plan (then IMG2D_SOURCE_REUSE does no forward step at all).  16
// bytes per position and step for two slots, against 8 L multiply-adds each way: streaming them costs
// less than the slab recomputation of the 16-slot kernel would.
//
// Transposed step.  out[y] = sum_k T_{row(y + M - k)}[k] V[y + M - k]: a gather by outputs would read
// another row for every tap.  Rows are read once, by the quad that owns their 8 input positions, and
// their products scattered: lane r's range of Q taps reaches outputs t = 0 ... Q + 6 of the block
// (output 8 b + t + s_r - M), accumulated over the 8 inputs in a sliding register window and stored to
// the array (r, t / 8), where every output position has exactly one writer; after a barrier each
// position sums its 4 ceil((Q + 7) / 8) entries in a fixed order.  No atomics, no exchange between
// quads.
//
// Measured on a B200: 5 shots of 500 x 250, 96 frequencies, 31 taps 5.61 -> 2.17 ms against the slab
// kernel of wlsq_adjoint.cuh; the L1 data pipe is 77% busy, half of it the shared-memory arrays.
#pragma once
#include "wlsq_adjoint.cuh"
#include "wlsq_rows.cuh"

namespace img2d {

constexpr int kRowsAdjX = 8;                  // input positions per quad in the transposed step
constexpr int kRowsAdjPos = 8 * kRowsAdjX;    // positions of one warp's transposed pass

template <int NS> struct RowsVec;
template <> struct RowsVec<1> { typedef float2 T; };
template <> struct RowsVec<2> { typedef float4 T; };

__host__ __device__ constexpr int rows_adj_arrays(int NP) { return (2 * NP + 7 + 7) / 8; }

__host__ __device__ inline int rows_adj_wp(int W) { return (W + kRowsAdjPos - 1) / kRowsAdjPos * kRowsAdjPos; }

// Entries of one scatter array: congruent 2 mod 8, so that the four lanes of two quads store to
// different banks.
__host__ __device__ inline int rows_adj_stride(int wp) { return (rows_pad(wp) + 7) / 8 * 8 + 2; }

__host__ __device__ inline size_t rows_adj_smem_bytes(int NS, int W, int L)
{
    const int wp = rows_adj_wp(W), left = ((L - 1) / 2 + 7) / 8 * 8;
    const size_t buf = rows_pad(left + wp + left) + 1;
    return (2 * buf + 4 * (size_t)rows_adj_arrays(rows_np(L)) * rows_adj_stride(wp)) * 8 * NS + 2 * (size_t)wp * 4 +
           (size_t)wp;
}

struct RowsAdjArgs {
    DemigrateArgs d;       // items, groups, geometry, index, source, reflectivity, data, counter, ckpt_mode
    const void *tab_rows;  // forward table in the row-split order
    int row_start[4], row_apart;
    void *planes;          // S_1 ... S_nextrap: [CTA or item][nextrap][plane] vectors of NS complex values
    long long plane;       // vectors per plane
};

template <int NS, int NP>
__global__ void __launch_bounds__(kRowsThreads, 1) demigrate_rows_kernel(RowsAdjArgs ra)
{
    typedef typename RowsVec<NS>::T Vec;
    constexpr int Q = 2 * NP, NF = (Q + 3) / 4, X = kRowsX, XB = kRowsAdjX, NA = rows_adj_arrays(NP);
    constexpr int ROWB = 64 * NP, C = 2 * NS;
    const DemigrateArgs &a = ra.d;
    const int M = a.M, L = 2 * M + 1;
    const int left = (M + 7) / 8 * 8;
    extern __shared__ float4 smem[];
    __shared__ int s_item;
    const int T = blockDim.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = T >> 5;
    const int r = lane & 3, qd = lane >> 3;
    const int p = (qd & (ra.row_apart - 1)) + ((lane >> 2) & 1) * ra.row_apart + (qd & -ra.row_apart) * 2;
    const char *tab = reinterpret_cast<const char *>(ra.tab_rows);
    const int tap0 = ra.row_start[r];
    const bool last_tap = tap0 + Q <= L;
    const int first_in = left - M + tap0 + (p * X & 7);
    const int hi8 = first_in >> 3, e8 = first_in & 7;

    auto load_taps = [&](RowTaps &o, unsigned off, int c) {
        if (Q - 4 * c >= 4) {
            rows_load8(o, tab + (size_t)(off + r * 32) + c * 128);
        } else {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(tab + (size_t)(off + r * 16) + c * 128));
            o.f[0] = v.x; o.f[1] = v.y; o.f[2] = v.z; o.f[3] = v.w;
        }
    };
    auto unpack = [&](const Vec &v, float (&f)[C]) {
        const float *q = reinterpret_cast<const float *>(&v);
#pragma unroll
        for (int e = 0; e < C; ++e) f[e] = q[e];
    };
    auto pack = [&](const float (&f)[C]) {
        Vec v;
        float *q = reinterpret_cast<float *>(&v);
#pragma unroll
        for (int e = 0; e < C; ++e) q[e] = f[e];
        return v;
    };
    auto mac = [&](float (&s)[C], float fr, float fi, const float (&v)[C]) {
#pragma unroll
        for (int g = 0; g < NS; ++g) {
            s[2 * g] = fmaf(fr, v[2 * g], s[2 * g]);
            s[2 * g + 1] = fmaf(fr, v[2 * g + 1], s[2 * g + 1]);
            s[2 * g] = fmaf(-fi, v[2 * g + 1], s[2 * g]);
            s[2 * g + 1] = fmaf(fi, v[2 * g], s[2 * g + 1]);
        }
    };

    for (;;) {
        if (threadIdx.x == 0) s_item = atomicAdd(a.counter, 1);
        __syncthreads();
        const int it = s_item;
        __syncthreads();
        if (it >= a.n_items) break;
        const int2 item = a.items[it];
        const GroupDesc grp = a.groups[item.x];
        const int j = item.y, u0 = grp.u0, W = grp.W;
        const int wp = rows_adj_wp(W), nwb = wp / kRowsWarpPos, nwb8 = wp / kRowsAdjPos;
        const int ns = rows_pad(left + wp + left) + 1, as = rows_adj_stride(wp);
        Vec *bufA = reinterpret_cast<Vec *>(smem), *bufB = bufA + ns, *arr = bufB + ns;
        unsigned *off0 = reinterpret_cast<unsigned *>(arr + (size_t)4 * NA * as), *off1 = off0 + wp;
        unsigned char *mask = reinterpret_cast<unsigned char *>(off1 + wp);  // bit g: slot g's shots cover x
        Vec *planes = reinterpret_cast<Vec *>(ra.planes) +
                      (long long)(a.ckpt_mode ? it : (int)blockIdx.x) * a.nextrap * ra.plane;
        {
            float zero[C] = {};
            for (int i = threadIdx.x; i < 2 * ns + 4 * NA * as; i += T) bufA[i] = pack(zero);
        }
        const uint16_t *idx_j = a.idx + (long long)j * a.idx_jstride;
        const int l0 = a.ckpt_mode == 2 ? a.nextrap - 1 : 0;  // first step to run
        for (int x = threadIdx.x; x < wp; x += T) {
            off0[x] = (unsigned)idx_j[(long long)l0 * a.idx_lstride + min(u0 + x, a.nx - 1)] * (unsigned)ROWB;
            unsigned m = 0;
            for (int g = 0; g < grp.nslots; ++g)
                if (x < W && a.owner[grp.owner_off + (long long)g * grp.owner_stride + x] >= 0) m |= 1u << g;
            mask[x] = (unsigned char)m;
        }
        __syncthreads();
        if (a.ckpt_mode != 2) {
            for (int k = grp.seg_begin; k < grp.seg_begin + grp.nseg; ++k) {
                const int4 sg = a.segs[k];
                const cpx *ws = a.wave + a.shot_off[sg.x] + (long long)j * sg.w;
                for (int i = threadIdx.x; i < sg.w; i += T) {
                    float *f = reinterpret_cast<float *>(bufA + rows_pad(left + sg.z - u0 + i)) + 2 * sg.y;
                    f[0] = ws[i].re;
                    f[1] = ws[i].im;
                }
            }
            __syncthreads();
        }

        // source: S_{l+1} = A_l S_l, every step kept
        for (int l = 0; a.ckpt_mode != 2 && l < a.nextrap; ++l) {
            const int ln = l + 1 < a.nextrap ? l + 1 : l;  // the first transposed step uses the last row again
            const uint16_t *inext = idx_j + (long long)ln * a.idx_lstride;
            Vec *keep = planes + (long long)l * ra.plane;
            for (int wb = warp; wb < nwb; wb += nwarps) {
                const int xb = (wb * 8 + p) * X;
                const unsigned nidx = inext[min(u0 + xb + r, a.nx - 1)];
                const uint4 o4 = *reinterpret_cast<const uint4 *>(off0 + xb);
                const unsigned off[X] = {o4.x, o4.y, o4.z, o4.w};
                const Vec *src = bufA + (hi8 + (xb >> 3)) * 9 + e8;
                float acc[X][C] = {};
                float win[X + 3][C];
                auto load_in = [&](int i, float (&v)[C]) {
                    unpack(src[((i & 7) >= 8 - e8 ? (i >> 3) + 1 : (i >> 3)) + i], v);
                };
#pragma unroll
                for (int i = 0; i < X - 1; ++i) load_in(i, win[i]);
#pragma unroll
                for (int c = 0; c < NF; ++c) {
                    const int nt = Q - 4 * c < 4 ? Q - 4 * c : 4;
                    RowTaps tp[X];
#pragma unroll
                    for (int jj = 0; jj < X; ++jj) load_taps(tp[jj], off[jj], c);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (i < nt) load_in(4 * c + X - 1 + i, win[X - 1 + i]);
#pragma unroll
                    for (int d = 0; d < 4; ++d) {
                        if (d < nt && (c < NF - 1 || d < nt - 1 || last_tap)) {
#pragma unroll
                            for (int jj = 0; jj < X; ++jj) mac(acc[jj], tp[jj].f[2 * d], tp[jj].f[2 * d + 1], win[jj + d]);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < X - 1; ++i)
#pragma unroll
                        for (int e = 0; e < C; ++e) win[i][e] = win[i + 4][e];
                }
                // reduce-scatter over the quad: lane r keeps output r
                const bool hi2 = (r & 2) != 0, hi1 = (r & 1) != 0;
                float out[C];
#pragma unroll
                for (int e = 0; e < C; ++e) {
                    float h[2];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const float keepv = hi2 ? acc[2 + i][e] : acc[i][e];
                        const float send = hi2 ? acc[i][e] : acc[2 + i][e];
                        h[i] = keepv + __shfl_xor_sync(0xffffffffu, send, 2);
                    }
                    const float keepv = hi1 ? h[1] : h[0], send = hi1 ? h[0] : h[1];
                    out[e] = keepv + __shfl_xor_sync(0xffffffffu, send, 1);
                }
                const unsigned m = mask[xb + r];
#pragma unroll
                for (int e = 0; e < C; ++e)
                    if (!((m >> (e / 2)) & 1u)) out[e] = 0.f;
                const Vec v = pack(out);
                bufB[rows_pad(left + xb + r)] = v;
                keep[xb + r] = v;
                off1[xb + r] = nidx * (unsigned)ROWB;
            }
            __syncthreads();
            Vec *t = bufA; bufA = bufB; bufB = t;
            unsigned *o = off0; off0 = off1; off1 = o;
        }

        // V_{nextrap-1} = m_{nextrap-1} S_nextrap
        for (int x = threadIdx.x; x < wp; x += T) {
            float s[C];
            unpack(planes[(long long)(a.nextrap - 1) * ra.plane + x], s);
            const float m = x < W ? a.refl[(long long)(a.nextrap - 1) * a.nx + u0 + x] : 0.f;
#pragma unroll
            for (int e = 0; e < C; ++e) s[e] *= m;
            bufA[rows_pad(left + x)] = pack(s);
        }
        __syncthreads();
        for (int l = a.nextrap - 1; l >= 0; --l) {
            const uint16_t *inext = idx_j + (long long)(l - 1) * a.idx_lstride;
            const Vec *Sl = planes + (long long)(l - 1) * ra.plane;
            const float *mrow = a.refl + (long long)(l - 1) * a.nx + u0;
            if (l > 0) {
                // what the emission after the barrier reads
                for (int x = threadIdx.x; x < W; x += T) {
                    if ((x & (128 / (int)sizeof(Vec) - 1)) == 0) asm volatile("prefetch.global.L1 [%0];" ::"l"(Sl + x));
                    if ((x & 31) == 0) asm volatile("prefetch.global.L1 [%0];" ::"l"(mrow + x));
                }
            }
            for (int wb = warp; wb < nwb8; wb += nwarps) {
                const int b = wb * 8 + p, xb = b * XB;
                const uint4 oa = *reinterpret_cast<const uint4 *>(off0 + xb), ob = *reinterpret_cast<const uint4 *>(off0 + xb + 4);
                const unsigned off[XB] = {oa.x, oa.y, oa.z, oa.w, ob.x, ob.y, ob.z, ob.w};
                const Vec *src = bufA + rows_pad(left + xb);
                Vec *dst = arr + (size_t)r * NA * as + 9 * b;
                float v[XB][C];
#pragma unroll
                for (int jj = 0; jj < XB; ++jj) unpack(src[jj], v[jj]);
                float acc[XB + 3][C] = {};
#pragma unroll
                for (int c = 0; c < NF; ++c) {
                    const int nt = Q - 4 * c < 4 ? Q - 4 * c : 4;
#pragma unroll
                    for (int jj = 0; jj < XB; ++jj) {
                        RowTaps tp;
                        load_taps(tp, off[jj], c);
#pragma unroll
                        for (int d = 0; d < 4; ++d) {
                            if (d >= nt) continue;
                            if (c < NF - 1 || d < nt - 1) {
                                mac(acc[jj + d], tp.f[2 * d], tp.f[2 * d + 1], v[jj]);
                            } else if (last_tap) {
                                mac(acc[jj + d], tp.f[2 * d], tp.f[2 * d + 1], v[jj]);
                            }
                        }
                    }
                    // the first nt outputs of the window have all their taps
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (i < nt) {
                            const int t = 4 * c + i;
                            dst[(size_t)(t >> 3) * as + (t & 7)] = pack(acc[i]);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < XB + 3; ++i)
#pragma unroll
                        for (int e = 0; e < C; ++e) acc[i][e] = i + nt < XB + 3 ? acc[i + nt][e] : 0.f;
                }
#pragma unroll
                for (int i = 0; i < XB - 1; ++i) {
                    const int t = Q + i;
                    dst[(size_t)(t >> 3) * as + (t & 7)] = pack(acc[i]);
                }
            }
            __syncthreads();
            for (int x = threadIdx.x; x < wp; x += T) {
                const unsigned nidx = l > 0 ? inext[min(u0 + x, a.nx - 1)] : 0u;
                float s[C] = {}, u[C] = {};
                float m = 0.f;
                if (l > 0 && x < W) {
                    unpack(Sl[x], s);  // zero outside the apertures
                    m = mrow[x];
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
#pragma unroll
                    for (int n = 0; n < NA; ++n) {
                        const int at = x + M - ra.row_start[q] - 8 * n;
                        if (at >= 0 && at < wp) {
                            float f[C];
                            unpack(arr[(size_t)(q * NA + n) * as + rows_pad(at)], f);
#pragma unroll
                            for (int e = 0; e < C; ++e) u[e] += f[e];
                        }
                    }
                }
                const unsigned in = mask[x];
#pragma unroll
                for (int e = 0; e < C; ++e) {
                    if (!((in >> (e / 2)) & 1u)) u[e] = 0.f;
                    if (l > 0) u[e] = fmaf(m, s[e], u[e]);
                }
                bufA[rows_pad(left + x)] = pack(u);
                off1[x] = nidx * (unsigned)ROWB;
            }
            __syncthreads();
            unsigned *o = off0; off0 = off1; off1 = o;
        }
        // bufA holds U_0 = F* m
        for (int k = grp.seg_begin; k < grp.seg_begin + grp.nseg; ++k) {
            const int4 sg = a.segs[k];
            cpx *ds = a.data + a.shot_off[sg.x] + (long long)j * sg.w;
            for (int i = threadIdx.x; i < sg.w; i += T) {
                const float *f = reinterpret_cast<const float *>(bufA + rows_pad(left + sg.z - u0 + i)) + 2 * sg.y;
                ds[i] = cpx{f[0], f[1]};
            }
        }
        __syncthreads();
    }
}

}  // namespace img2d
