// Front end of the migration: source wavelets and frequency-domain records on the device.
//
// Reference (file:line within the reference project ahadji05/Imaging2D_WLSQ):
//   main.py:111-123           per shot: Ricker source wavelet sampled on (nt, nx), receiver record read
//                             from CSV, both transformed along time with scipy.fftpack.fft (axis 0);
//                             the extrapolation then uses the first nw frequency rows
//   py_src/operatorsPreparation/util.py:10-14   ricker_wv_map(t) = (1 - 2 pi^2 f^2 t^2) exp(-pi^2 f^2 t^2),
//                             f = 30 Hz
//   py_src/operatorsPreparation/util.py:47-58   makeRickerWavelet: r = sqrt((init_depth - isz)^2 +
//                             (xi - sx)^2), t0 = r / v, t_t0 = tj - t0 stored as float32, wavelet[j, i] =
//                             ricker(t_t0[j]) / sqrt(r), accumulated into a float32 array
//
// The transform along time keeps nf of nt rows and every trace is a column of its own, so a library
// transform computes rows that nobody reads and writes them to memory for a packing pass.  The two
// kernels below write the kept rows straight into the packed layout:
//   records  record_spectra_kernel, a two-stage transform nt = N1 x N2 of 16 (or 8) traces per CTA in
//            shared memory, single precision like the reference's transform of float32 records;
//   sources  source_spectra_kernel: a Ricker wavelet sampled in float32 is exactly zero away from its
//            arrival, so its spectrum is a short sum and the time-domain array is never formed.
// Lengths without a divisor that makes the first worthwhile (primes), and most rows of many large
// records, go through cuFFT, one
// real-to-complex transform per shot, and pack_spectra_kernel.
//
// Measured on a B200, 32 shots of 1500 x 1024 samples, 256 rows, sources and records: 2.33 ms with
// cuFFT (64 transforms, a wavelet array of 0.2 GB), 0.45 ms now: 0.28 ms for the records (58% of the
// issue slots, 39% of the FMA pipe; the reads alone would take 0.03 ms) and 0.13 ms for the sources.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "wlsq_kernels.cuh"

namespace img2d {

// out[s][j][i] (float32, time domain) for ns sources at sx[s] (model x in metres).
__global__ void ricker_sources_kernel(int ns, int nt, int nx, double dt, double x_first, double dx, double dzr,
                                      double v, double fpeak, const double *__restrict__ sx,
                                      float *__restrict__ out)
{
    const long long total = (long long)ns * nt * nx;
    const double pf2 = 9.869604401089358 * fpeak * fpeak;  // pi^2 f^2
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(e % nx);
        const long long r0 = e / nx;
        const int j = (int)(r0 % nt);
        const int s = (int)(r0 / nt);
        const double xi = x_first + i * dx;
        const double ddx = xi - sx[s];
        const double r = sqrt(dzr * dzr + ddx * ddx);
        const float tt = (float)((double)j * dt - r / v);  // the reference keeps t - t0 in float32
        const double term = pf2 * (double)tt * (double)tt;
        out[e] = (float)((1.0 - 2.0 * term) * exp(-term) / sqrt(r));
    }
}

// Packs the first nf rows of real-to-complex spectra into the migration's per-shot aperture layout.
// spec: (nsc, nt/2+1, nx) complex, the transforms along time of shots s0 .. s0+nsc-1; row j of the
// full spectrum is spec row j for j <= nt/2 and conj(spec row nt-j) above (real input).
// out: shot s's block at off[s], row j, column x - x0[s] for x in [x0[s], x0[s] + w[s]).
__global__ void pack_spectra_kernel(int s0, int nsc, int nt, int nx, int nf, const cpx *__restrict__ spec,
                                    const int *__restrict__ x0, const int *__restrict__ w,
                                    const long long *__restrict__ off, cpx *__restrict__ out)
{
    const int nh = nt / 2 + 1;
    const long long total = (long long)nsc * nf * nx;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(e % nx);
        const long long r = e / nx;
        const int j = (int)(r % nf);
        const int sl = (int)(r / nf);
        const int s = s0 + sl;
        const int xs = x0[s], ws = w[s];
        if (x < xs || x >= xs + ws) continue;
        cpx v;
        if (j < nh) {
            v = spec[((long long)sl * nh + j) * nx + x];
        } else {
            const cpx c = spec[((long long)sl * nh + (nt - j)) * nx + x];
            v = cpx{c.re, -c.im};
        }
        out[off[s] + (long long)j * ws + (x - xs)] = v;
    }
}

// Up to kSpecShots shots of one launch, passed by value: no upload, no device allocation.
constexpr int kSpecShots = 64;
struct SpecShots {
    int x0[kSpecShots], w[kSpecShots];
    long long off[kSpecShots];
    double sx[kSpecShots];  // source positions (source_spectra_kernel)
};

// exp(-2 pi i m / n), evaluated in double and rounded once
__device__ __forceinline__ float2 unit_root(long long m, int n)
{
    double sn, cs;
    sincospi(-2.0 * (double)(m % n) / (double)n, &sn, &cs);
    return make_float2((float)cs, (float)sn);
}

// Two-stage transform X[k] = sum_{t2 < N2} e(t2 k / nt) sum_{t1 < N1} x[N2 t1 + t2] e(t1 k / N1),
// e(y) = exp(-2 pi i y).  The inner sums depend on k mod N1 and, for real input, come in conjugate
// pairs: K1 = N1/2 + 1 of them are formed per t2.
//
// Tables: T1[t][kSpecK] (cos, sin)(2 pi t k1 / N1) for t <= N1/2, k1 < kSpecK; the outer factor
// e(t2 (k1 + N1 m) / nt) as A[k1][t2] = e(t2 k1 / nt) times B[t2][mp] = e(t2 m / N2), m < mp.
constexpr int kSpecK = 16;    // inner outputs: N1 <= 31
constexpr int kSpecKC = 8;    // of them per task
constexpr int kSpecT = 4;     // values of t2 per task
constexpr int kSpecBlock = 8; // terms of a partial sum of the second stage
struct SpecPlan {
    int N1, N2, K1, mp, C, M;  // C: traces per CTA, M: outer outputs per thread and pass
    int S, T2;                     // second stage: parts of the sum over t2 (1: whole sums), terms of a part
    bool bs;                       // table B in shared memory
    size_t smem;
};

__global__ void spec_tables_kernel(SpecPlan pl, int nt, float2 *__restrict__ T1, float2 *__restrict__ B,
                                   float2 *__restrict__ A)
{
    const int n1 = kSpecK * kSpecK, n2 = pl.N2 * pl.mp;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n1 + n2 + nt; e += gridDim.x * blockDim.x) {
        if (e < n1) {
            const float2 c = unit_root((long long)(e / kSpecK) * (e % kSpecK), pl.N1);
            T1[e] = make_float2(c.x, -c.y);
        } else if (e < n1 + n2) {
            B[e - n1] = unit_root((long long)((e - n1) / pl.mp) * ((e - n1) % pl.mp), pl.N2);
        } else {
            const int i = e - n1 - n2;
            A[i] = unit_root((long long)(i % pl.N2) * (i / pl.N2), nt);
        }
    }
}

// One CTA: C traces of one shot.  Both stages are small matrix products whose factors (the tables) are
// the same for all lanes; a 16-byte load of them costs four cycles of the L1 write-back however few
// addresses it has, so each must feed many multiply-adds:
//   stage 1  a task is C traces, four values of t2 and 8 inner outputs; real sums over
//            x[t] + x[N1 - t] and x[t] - x[N1 - t] (half the multiply-adds): 16 per load;
//   stage 2  a task is C traces, two per thread, and M outputs k1 + N1 m of one residue k1: 16 per
//            load; the inner sum is turned by A once and B, common to the residues, sits in shared
//            memory (BS, up to 8 KB: one load from L2 per factor was waited for 50 times).  Sums of 8 terms, then their sum: with one running sum over N2 = 50 terms the error
//            against 64 bits was 2.1e-7, cuFFT's 1.6e-7.
// One trace per thread and 8 per load: 446 us for 32 shots of 1500 x 1024 samples, 256 rows.
// SPLIT: lengths with few residues (a large prime times 1 to 4) have a few tasks of very long sums.  Their
// sums over t2 are shared out over the idle threads in S parts, added in order at the end: 25
// shots of 1553 x 716 samples, 20 rows, with their sources 4.0 ms without, 0.42 with (cuFFT 0.73).
template <int C, int M, bool BS, bool SPLIT>
__global__ void __launch_bounds__(256, 2) record_spectra_kernel(SpecPlan pl, SpecShots sh, int s0, int nt, int nx,
                                                                int nf, const float *__restrict__ rec,
                                                                const float2 *__restrict__ T1,
                                                                const float2 *__restrict__ B,
                                                                const float2 *__restrict__ A, cpx *__restrict__ out)
{
    extern __shared__ float4 spec_smem[];
    float4 *const Bs = spec_smem;  // BS: B
    float2 *const Y = reinterpret_cast<float2 *>(spec_smem + (BS ? pl.N2 * pl.mp / 2 : 0));  // [t2][k1][C]
    __shared__ float4 tw[kSpecK * kSpecK / 2];
    const int sl = blockIdx.y, x0 = blockIdx.x * C;
    const int xs = sh.x0[sl], ws = sh.w[sl];
    if (x0 + C <= xs || x0 >= xs + ws) return;  // no trace of the aperture
    const int N1 = pl.N1, N2 = pl.N2, K1 = pl.K1;
    for (int i = threadIdx.x; i < kSpecK * kSpecK / 2; i += 256) tw[i] = reinterpret_cast<const float4 *>(T1)[i];
    if (BS)
        for (int i = threadIdx.x; i < N2 * pl.mp / 2; i += 256) Bs[i] = reinterpret_cast<const float4 *>(B)[i];
    __syncthreads();
    {
        const int col = threadIdx.x % C, nq = (N2 + kSpecT - 1) / kSpecT;
        const float *xr = rec + (long long)(s0 + sl) * nt * nx + min(x0 + col, nx - 1);
        const long long st1 = (long long)N2 * nx;
        for (int task = threadIdx.x / C; task < nq * ((K1 + kSpecKC - 1) / kSpecKC); task += 256 / C) {
            const int ta = task % nq * kSpecT, kc = task / nq * kSpecKC;
            const float *px[kSpecT];
            float re[kSpecT][kSpecKC], im[kSpecT][kSpecKC];
#pragma unroll
            for (int i = 0; i < kSpecT; ++i) {
                px[i] = xr + (long long)min(ta + i, N2 - 1) * nx;
                const float v = px[i][0];
#pragma unroll
                for (int k = 0; k < kSpecKC; ++k) {
                    re[i][k] = v;
                    im[i][k] = 0.f;
                }
            }
#pragma unroll 4
            for (int t = 1; 2 * t <= N1; ++t) {
                const bool mid = 2 * t == N1;
                float s[kSpecT], d[kSpecT];
#pragma unroll
                for (int i = 0; i < kSpecT; ++i) {
                    const float u = px[i][t * st1], v = mid ? 0.f : px[i][(N1 - t) * st1];
                    s[i] = u + v;
                    d[i] = mid ? 0.f : v - u;
                }
#pragma unroll
                for (int k = 0; k < kSpecKC; k += 2) {
                    const float4 c = tw[(t * kSpecK + kc + k) / 2];  // cos, sin of k and k + 1
#pragma unroll
                    for (int i = 0; i < kSpecT; ++i) {
                        re[i][k] = fmaf(s[i], c.x, re[i][k]);
                        im[i][k] = fmaf(d[i], c.y, im[i][k]);
                        re[i][k + 1] = fmaf(s[i], c.z, re[i][k + 1]);
                        im[i][k + 1] = fmaf(d[i], c.w, im[i][k + 1]);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < kSpecT; ++i)
#pragma unroll
                for (int k = 0; k < kSpecKC; ++k)
                    if (kc + k < K1 && ta + i < N2)
                        Y[((ta + i) * K1 + kc + k) * C + col] = make_float2(re[i][k], im[i][k]);
        }
    }
    __syncthreads();
    constexpr int H = C / 2;  // threads per task; traces col and col + H
    const int col = threadIdx.x % H;
    const int nm = pl.mp / M, tasks = min(N1, nf) * nm;
    // sums of outputs k1 + N1 (m0 + m) over t2 in [first, last)
    auto sum = [&](int k1, int m0, int first, int last, float (&sre)[2][M], float (&sim)[2][M]) {
        const bool conj = k1 >= K1;
        const float2 *y = Y + (conj ? N1 - k1 : k1) * C + col;
        const float4 *w = BS ? Bs + m0 / 2 : reinterpret_cast<const float4 *>(B + m0);
        const float2 *turn = A + (long long)k1 * N2;
#pragma unroll
        for (int m = 0; m < M; ++m) sre[0][m] = sim[0][m] = sre[1][m] = sim[1][m] = 0.f;
        for (int tb = first; tb < last; tb += kSpecBlock) {
            float re[2][M], im[2][M];
#pragma unroll
            for (int m = 0; m < M; ++m) re[0][m] = im[0][m] = re[1][m] = im[1][m] = 0.f;
#pragma unroll 2
            for (int t2 = tb; t2 < min(tb + kSpecBlock, last); ++t2) {
                float2 v[2] = {y[t2 * K1 * C], y[t2 * K1 * C + H]};
                const float2 q = __ldg(turn + t2);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float vr = v[i].x, vi = conj ? -v[i].y : v[i].y;
                    v[i].x = fmaf(vr, q.x, -vi * q.y);
                    v[i].y = fmaf(vr, q.y, vi * q.x);
                }
#pragma unroll
                for (int m = 0; m < M; m += 2) {
                    const float4 c = BS ? w[(t2 * pl.mp + m) / 2] : __ldg(w + (t2 * pl.mp + m) / 2);
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        re[i][m] = fmaf(v[i].x, c.x, re[i][m]);
                        im[i][m] = fmaf(v[i].x, c.y, im[i][m]);
                        re[i][m] = fmaf(-v[i].y, c.y, re[i][m]);
                        im[i][m] = fmaf(v[i].y, c.x, im[i][m]);
                        re[i][m + 1] = fmaf(v[i].x, c.z, re[i][m + 1]);
                        im[i][m + 1] = fmaf(v[i].x, c.w, im[i][m + 1]);
                        re[i][m + 1] = fmaf(-v[i].y, c.w, re[i][m + 1]);
                        im[i][m + 1] = fmaf(v[i].y, c.z, im[i][m + 1]);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int m = 0; m < M; ++m) {
                    sre[i][m] += re[i][m];
                    sim[i][m] += im[i][m];
                }
        }
    };
    auto store = [&](int k1, int m0, const float (&sre)[2][M], const float (&sim)[2][M]) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int x = x0 + col + i * H;
            if (x < xs || x >= xs + ws) continue;
            cpx *o = out + sh.off[sl] + (x - xs);
#pragma unroll
            for (int m = 0; m < M; ++m) {
                const int k = k1 + N1 * (m0 + m);
                if (k < nf) o[(long long)k * ws] = cpx{sre[i][m], sim[i][m]};
            }
        }
    };
    float sre[2][M], sim[2][M];
    if (!SPLIT) {
        for (int task = threadIdx.x / H; task < tasks; task += 256 / H) {
            const int k1 = task / nm, m0 = task % nm * M;
            if (k1 + N1 * m0 >= nf) continue;
            sum(k1, m0, 0, N2, sre, sim);
            store(k1, m0, sre, sim);
        }
        return;
    }
    // S tasks <= 256 / H: one part a thread
    const int part = threadIdx.x / H / tasks, task = threadIdx.x / H % tasks;
    const int k1 = task / nm, m0 = task % nm * M;
    const bool active = part < pl.S && k1 + N1 * m0 < nf;
    if (active) sum(k1, m0, part * pl.T2, min((part + 1) * pl.T2, N2), sre, sim);
    __syncthreads();
    float2 *const P = Y;  // [part][task][2 M][H], once Y has been read
    if (active && part > 0) {
#pragma unroll
        for (int e = 0; e < 2 * M; ++e)
            P[((part * tasks + task) * 2 * M + e) * H + col] = make_float2(sre[e / M][e % M], sim[e / M][e % M]);
    }
    __syncthreads();
    if (active && part == 0) {
        for (int r = 1; r < pl.S; ++r) {
#pragma unroll
            for (int e = 0; e < 2 * M; ++e) {
                const float2 v = P[((r * tasks + task) * 2 * M + e) * H + col];
                sre[e / M][e % M] += v.x;
                sim[e / M][e % M] += v.y;
            }
        }
        store(k1, m0, sre, sim);
    }
}

// Sources: spectrum of the sampled wavelet of ricker_sources_kernel.  Past |t - t0| = tw its value is
// zero in float32 (tw is chosen so that the exponent exceeds 150), so rows jlo ... jlo + nsup - 1 of
// the column are summed, exp(-2 pi i j k / nt) as exp(-2 pi i jlo k / nt) exp(-2 pi i n k / nt): the
// second factor is the same for all columns (U[n][kp], k along rows).
constexpr int kSrcK = 8;
__global__ void source_tables_kernel(int nt, int nw, int nsup, int kp, float2 *__restrict__ W,
                                     float2 *__restrict__ U)
{
    for (long long e = blockIdx.x * blockDim.x + threadIdx.x; e < nw + (long long)nsup * kp;
         e += gridDim.x * blockDim.x) {
        if (e < nw) W[e] = unit_root(e, nt);
        else U[e - nw] = unit_root((e - nw) / kp * ((e - nw) % kp), nt);
    }
}

// One CTA: kSrcCols columns of one shot; a thread sums kSrcK rows of four columns, 16 multiply-adds per
// 16-byte load of U (with one column per thread the loads' write-back took four times the arithmetic).
constexpr int kSrcCols = 128;
__global__ void __launch_bounds__(256) source_spectra_kernel(SpecShots sh, int nt, int nx, int nf, int nsup, int kp,
                                                             double dt, double x_first, double dx, double dzr,
                                                             double v, double fpeak, double tw,
                                                             const float2 *__restrict__ W,
                                                             const float2 *__restrict__ U, cpx *__restrict__ out)
{
    constexpr int NC = kSrcCols / 32;
    extern __shared__ float wav[];  // [nsup][kSrcCols]
    __shared__ int first_row[kSrcCols];
    __shared__ double arrival[kSrcCols], amp[kSrcCols];
    const int sl = blockIdx.y, x0 = blockIdx.x * kSrcCols;
    const int xs = sh.x0[sl], ws = sh.w[sl];
    if (x0 + kSrcCols <= xs || x0 >= xs + ws) return;
    const double pf2 = 9.869604401089358 * fpeak * fpeak;  // pi^2 f^2
    if (threadIdx.x < kSrcCols) {
        const double ddx = x_first + (x0 + (int)threadIdx.x) * dx - sh.sx[sl];
        const double r = sqrt(dzr * dzr + ddx * ddx), t0 = r / v;
        const double first = floor((t0 - tw) / dt);
        arrival[threadIdx.x] = t0;
        amp[threadIdx.x] = sqrt(r);
        first_row[threadIdx.x] = first > 0.0 ? (first < (double)nt ? (int)first : nt) : 0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nsup * kSrcCols; i += 256) {
        const int n = i / kSrcCols, c = i % kSrcCols, j = first_row[c] + n;
        float val = 0.f;
        if (j < nt) {
            const float tt = (float)((double)j * dt - arrival[c]);  // the reference keeps t - t0 in float32
            const double term = pf2 * (double)tt * (double)tt;
            val = (float)((1.0 - 2.0 * term) * exp(-term) / amp[c]);
        }
        wav[i] = val;
    }
    __syncthreads();
    const int col = threadIdx.x & 31, part = threadIdx.x >> 5;
    for (int k0 = (blockIdx.z * 8 + part) * kSrcK; k0 < nf; k0 += gridDim.z * 8 * kSrcK) {
        const float4 *u = reinterpret_cast<const float4 *>(U + k0);
        float re[NC][kSrcK], im[NC][kSrcK];
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int k = 0; k < kSrcK; ++k) re[c][k] = im[c][k] = 0.f;
#pragma unroll 4
        for (int n = 0; n < nsup; ++n) {
            float w[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) w[c] = wav[n * kSrcCols + col + 32 * c];
#pragma unroll
            for (int k = 0; k < kSrcK; k += 2) {
                const float4 q = __ldg(u + (n * kp + k) / 2);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    re[c][k] = fmaf(w[c], q.x, re[c][k]);
                    im[c][k] = fmaf(w[c], q.y, im[c][k]);
                    re[c][k + 1] = fmaf(w[c], q.z, re[c][k + 1]);
                    im[c][k + 1] = fmaf(w[c], q.w, im[c][k + 1]);
                }
            }
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int x = x0 + col + 32 * c;
            if (x < xs || x >= xs + ws) continue;
            cpx *o = out + sh.off[sl] + (x - xs);
            const int jlo = min(first_row[col + 32 * c], nt - 1);
            int at = (int)((long long)jlo * k0 % nt);  // jlo k mod nt
#pragma unroll
            for (int k = 0; k < kSrcK; ++k) {
                if (k0 + k >= nf) continue;
                const float2 ph = __ldg(W + at);
                at += jlo;
                if (at >= nt) at -= nt;
                o[(long long)(k0 + k) * ws] =
                    cpx{fmaf(re[c][k], ph.x, -im[c][k] * ph.y), fmaf(re[c][k], ph.y, im[c][k] * ph.x)};
            }
        }
    }
}

}  // namespace img2d
