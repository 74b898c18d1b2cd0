// tdf_kernels.cuh -- the hot-path kernels of the job_core() chain
// (search/network/openmp/jobcore.c:193-630) other than the FFT passes:
//
//   sky stage (FP64, once per sky point and detector): tdf_sky.cuh
//   injection: k_signal, k_add_signal
//   spindown stage (once per template)
//     (the passes: tdf_split.cuh)
//     DemodSplit      column-pass prologue of the allocation-free entry point:
//                     spindown_modulation (spinmod.c:490-514)
//     StoreFstat      its row-pass epilogue: F = |Fa|^2/aa + |Fb|^2/bb
//                     (jobcore.c:481-484)
//     k_block_means   FStat blocks_avg means (auxi.c:336-363)
//     k_threshold     MAX_ALG 3 local maxima, veto, trigger append
//                     (jobcore.c:552-603)
#pragma once

#include <float.h>
#include <math_constants.h>

#include <type_traits>

#include "tdf_bulk.cuh"
#include "tdf_passes.cuh"

namespace tdf {

struct SkyParam {
     double sinalt, cosalt, sindelt, cosdelt, het0;
     double nS0, nS1, nS2;
};

struct DetParam {
     double amod[9];
     double cphir, sphir, sig2;
};

// one template: (sky slot, spindown)
struct TmplParam {
     double het1;     // fmod(ss*M[4], M[0]) (+M[0] if negative), FP64
     double spnd;     // ss*M[5] + nn*M[9] + mm*M[13], FP64
     double sgnl0;    // het0 + het1 as the emulated build rounds it (trigger frequency)
     int32_t slot;    // operand slot of the sky point
     uint32_t id;     // template number within the call
};

struct AaBb {
     double aa, bb;
     float aaf, bbf;
};

struct Trig {
     uint32_t id, bin;
     float f, F;
};

constexpr unsigned ERR_OVERFLOW = 1u;
constexpr double TWO_PI = 6.283185307179586476925286766559;
constexpr double INV_TWO_PI = 0.15915494309189533576888376337251;
constexpr double M_PI_D = 3.14159265358979323846;

// ------------------------------------------------------------------ sky stage

// modvir (settings.c:254-294) at one sample: the amplitude modulations
// a(t), b(t) of detector D for a source at (alpha, delta), 0 where
// |xDat[t]| <= DBL_MIN
__device__ __forceinline__ void modvir_at(const DetParam &D, double sinal, double cosal, double sindel, double cosdel,
                                          double cosm, double sinm, float x, double &aa, double &bb) {
     const double cosalfr = cosal * D.cphir + sinal * D.sphir;
     const double sinalfr = sinal * D.cphir - cosal * D.sphir;
     const double c2d = cosdel * cosdel, c2sd = sindel * cosdel;
     const double c = cosalfr * cosm + sinalfr * sinm;
     const double s = sinalfr * cosm - cosalfr * sinm;
     const double c2s = 2. * c * c, cs = c * s;
     const bool on = fabs((double)x) > DBL_MIN;
     aa = D.amod[0] * (2. - c2d) * c2s + D.amod[1] * (2. - c2d) * 2. * cs +
          D.amod[2] * c2sd * c + D.amod[3] * c2sd * s - D.amod[0] * (2. - c2d) + D.amod[4] * c2d;
     bb = D.amod[5] * sindel * c2s + D.amod[6] * sindel * 2. * cs +
          D.amod[7] * cosdel * c + D.amod[8] * cosdel * s - D.amod[5] * sindel;
     aa = on ? aa : 0.;
     bb = on ? bb : 0.;
}

// ------------------------------------------------------------------ injection

// add_signal (init.c:365-504) constants, formed on the host in the
// reference's evaluation order
struct SignalParam {
     double sinal, cosal, sindel, cosdel;   // of the source
     double nS0, nS1, nS2;                  // cos a cos d, sin a cos d, sin d
     double amp[4];                         // amplit[] (init.c:411-414)
     double freqo0, freqo1, phaseshift;     // init.c:382-386, 417-418
     double dephase;                        // 2 pi dt fpo (init.c:447)
};

// grid (ceil(N/256), nifo), 256 threads: the signal s_n[i] of detector n
// (init.c:428-456) into s[n*N + i], and per-block sums of s^2 into
// partial[n*gridDim.x + block].  Products and sums are not contracted, as
// in the reference's DOUBLE build (the phase reaches ~1e8 rad).
__global__ void __launch_bounds__(256) k_signal(
     const float *__restrict__ xdat, const double *__restrict__ detssb, const double *__restrict__ cosm,
     const double *__restrict__ sinm, const DetParam *__restrict__ dp, int N, int Nal, SignalParam P,
     double *__restrict__ s, double *__restrict__ partial)
{
     const int d = blockIdx.y;
     const int i = blockIdx.x * 256 + threadIdx.x;
     double v = 0.;
     if (i < N) {
          const DetParam &D = dp[d];
          double aa, bb;
          modvir_at(D, P.sinal, P.cosal, P.sindel, P.cosdel, cosm[i], sinm[i], xdat[(size_t)d * Nal + i], aa, bb);
          const double *e = detssb + (size_t)d * 3 * N + 3 * (size_t)i;
          const double sh = __dadd_rn(__dadd_rn(__dmul_rn(P.nS0, e[0]), __dmul_rn(P.nS1, e[1])), __dmul_rn(P.nS2, e[2]));
          const double di = (double)i;
          // freqo0*(i + sh) + freqo1*(2 sh i + i^2 + sh^2) + phaseshift - dephase*i
          const double q = __dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(2., sh), di), __dmul_rn(di, di)), __dmul_rn(sh, sh));
          double ph = __dadd_rn(__dadd_rn(__dmul_rn(P.freqo0, __dadd_rn(di, sh)), __dmul_rn(P.freqo1, q)), P.phaseshift);
          ph = __dsub_rn(ph, __dmul_rn(P.dephase, di));
          double sn, cn;
          sincos(ph, &sn, &cn);
          v = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(P.amp[0], aa), cn), __dmul_rn(__dmul_rn(P.amp[1], bb), cn)),
                                  __dmul_rn(__dmul_rn(P.amp[2], aa), sn)),
                        __dmul_rn(__dmul_rn(P.amp[3], bb), sn));
          s[(size_t)d * N + i] = v;
     }
     double v2 = v * v;
#pragma unroll
     for (int o = 16; o > 0; o >>= 1) v2 += __shfl_down_sync(0xffffffffu, v2, o);
     __shared__ double red[8];
     if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v2;
     __syncthreads();
     if (threadIdx.x == 0) {
          double t = 0.;
          for (int k = 0; k < 8; k++) t += red[k];
          partial[(size_t)d * gridDim.x + blockIdx.x] = t;
     }
}

// grid (ceil(N/256), nifo), 256 threads: xDat[i] += h0 s_n[i] where xDat[i]
// != 0, the sum in FP64 and rounded to float once (init.c:468-473)
__global__ void __launch_bounds__(256) k_add_signal(float *__restrict__ xdat, const double *__restrict__ s, int N,
                                                    int Nal, double h0)
{
     const int d = blockIdx.y;
     const int i = blockIdx.x * 256 + threadIdx.x;
     if (i >= N) return;
     float *x = xdat + (size_t)d * Nal + i;
     if (*x != 0.f) *x = (float)__dadd_rn((double)*x, __dmul_rn(h0, s[(size_t)d * N + i]));
}

// ------------------------------------------------------------------ spindown stage

// Neumaier-compensated accumulation of the detector-network sum
struct CompSum {
     float s, c;
     __device__ __forceinline__ void init(float v) { s = v; c = 0.f; }
     __device__ __forceinline__ void add(float x) {
          float t = s + x;
          c += (fabsf(s) >= fabsf(x)) ? ((s - t) + x) : ((x - t) + s);
          s = t;
     }
     __device__ __forceinline__ float value() const { return s + c; }
};

// Split form: phase = het1*i + spnd*i^2 formed and reduced mod 2 pi in FP64,
// plus spnd*(2 i shft_n[i]) in FP32 per detector; FP32 sincos and products.
// The detector-network sum is compensated (Neumaier) for three or more
// detectors; for one or two it is a single rounded addition, which the
// compensation would not change.  Operands planar by detector,
// xab[(slot*nifo + d)*Nal + i] (the layout tdf_fstat_operands_static takes).
struct DemodSplit {
     const float4 *xab;
     const float *s2;
     const TmplParam *tp;
     int N, N2, Nal, nifo;
     static constexpr int kQ = 1;   // elements whose operand loads are issued together

     // x * (cs - i sn) for the two arrays of an operand x = (a.re, a.im, b.re, b.im)
     static __device__ __forceinline__ void rot(const float4 x, float phf, float2 &pa, float2 &pb) {
          float sn, cs;
          __sincosf(phf, &sn, &cs);
          pa = make_float2(fmaf(x.x, cs, x.y * sn), fmaf(x.y, cs, -x.x * sn));
          pb = make_float2(fmaf(x.z, cs, x.w * sn), fmaf(x.w, cs, -x.z * sn));
     }

     template <int L>
     __device__ __forceinline__ void load(float2 (&v)[2][8], int b, int n2, int t) const {
          const TmplParam P = tp[b];
          const float spf = (float)P.spnd;
          const size_t base = (size_t)P.slot * nifo * Nal;
#pragma unroll
          for (int h = 0; h < 8 / kQ; h++) {
               int ii[kQ];
               float pr[kQ];
#pragma unroll
               for (int q = 0; q < kQ; q++) ii[q] = N2 * (t + (kQ * h + q) * (L / 8)) + n2;
               float2 fa[kQ], fb[kQ];
               if (ii[0] >= N) {
                    // zero padding beyond N: the whole group (the tail rows of
                    // every column, uniform across the warp)
#pragma unroll
                    for (int q = 0; q < kQ; q++) {
                         v[0][kQ * h + q] = make_float2(0.f, 0.f);
                         v[1][kQ * h + q] = make_float2(0.f, 0.f);
                    }
                    continue;
               }
#pragma unroll
               for (int q = 0; q < kQ; q++) {
                    const double di = (double)ii[q];
                    const double ph = fma(P.spnd, di * di, P.het1 * di);
                    const double kk = rint(ph * INV_TWO_PI);
                    pr[q] = (float)fma(-kk, TWO_PI, ph);
               }
               if (nifo <= 2) {
                    float4 x0[kQ], x1[kQ];
                    float s0[kQ], s1[kQ];
#pragma unroll
                    for (int q = 0; q < kQ; q++) {
                         const bool ok = ii[q] < N;
                         const size_t o = base + ii[q];
                         x0[q] = ok ? __ldg(&xab[o]) : make_float4(0.f, 0.f, 0.f, 0.f);
                         s0[q] = ok ? __ldg(&s2[o]) : 0.f;
                         const bool ok1 = ok && nifo == 2;
                         x1[q] = ok1 ? __ldg(&xab[o + Nal]) : make_float4(0.f, 0.f, 0.f, 0.f);
                         s1[q] = ok1 ? __ldg(&s2[o + Nal]) : 0.f;
                    }
#pragma unroll
                    for (int q = 0; q < kQ; q++) {
                         if (ii[q] >= N) {
                              fa[q] = make_float2(0.f, 0.f);
                              fb[q] = make_float2(0.f, 0.f);
                              continue;
                         }
                         rot(x0[q], fmaf(spf, s0[q], pr[q]), fa[q], fb[q]);
                         if (nifo == 2) {
                              float2 pa, pb;
                              rot(x1[q], fmaf(spf, s1[q], pr[q]), pa, pb);
                              fa[q] = cadd(fa[q], pa);
                              fb[q] = cadd(fb[q], pb);
                         }
                    }
               } else {
#pragma unroll
                    for (int q = 0; q < kQ; q++) {
                         fa[q] = make_float2(0.f, 0.f);
                         fb[q] = make_float2(0.f, 0.f);
                         if (ii[q] >= N) continue;
                         CompSum ar, ai, br, bi;
                         for (int d = 0; d < nifo; d++) {
                              const size_t o = base + (size_t)d * Nal + ii[q];
                              float2 pa, pb;
                              rot(__ldg(&xab[o]), fmaf(spf, __ldg(&s2[o]), pr[q]), pa, pb);
                              if (d == 0) { ar.init(pa.x); ai.init(pa.y); br.init(pb.x); bi.init(pb.y); }
                              else { ar.add(pa.x); ai.add(pa.y); br.add(pb.x); bi.add(pb.y); }
                         }
                         fa[q] = make_float2(ar.value(), ai.value());
                         fb[q] = make_float2(br.value(), bi.value());
                    }
               }
#pragma unroll
               for (int q = 0; q < kQ; q++) {
                    v[0][kQ * h + q] = fa[q];
                    v[1][kQ * h + q] = fb[q];
               }
          }
     }
};

// Row-pass epilogue of the allocation-free entry point: F[k] over [fr0, fr1].
struct StoreFstat {
     float *F;
     const TmplParam *tp;
     const AaBb *ab;
     int nF, fr0, fr1, N1;
     template <int L>
     __device__ __forceinline__ void store(const float2 (&v)[2][8], int b, int k1, int t) const {
          const AaBb s = ab[tp[b].slot];
          float *dst = F + (size_t)b * nF - fr0;
#pragma unroll
          for (int m = 0; m < 8; m++) {
               const int k = k1 + N1 * (t + m * (L / 8));
               if (k >= fr0 && k <= fr1) dst[k] = cnorm(v[0][m]) / s.aaf + cnorm(v[1][m]) / s.bbf;
          }
     }
};

}  // namespace tdf

#include "tdf_split.cuh"
#include "tdf_sky.cuh"

namespace tdf {

// blocks_avg means (auxi.c:349-355): mu_j = sum of the j-th block of NAV
// values of F[fr0..] / (2 NAV).  grid (nblk, ntmpl), 256 threads
template <typename T>
__global__ void k_block_means(const T *__restrict__ F, int nF, int nblk, T *__restrict__ mu)
{
     const int j = blockIdx.x, b = blockIdx.y;
     const T *src = F + (size_t)b * nF + (size_t)j * 4096;
     T v[16], s = 0;
#pragma unroll
     for (int k = 0; k < 16; k++) v[k] = src[threadIdx.x + 256 * k];   // all in flight
#pragma unroll
     for (int k = 0; k < 16; k++) s += v[k];
     __shared__ T red[256];
     red[threadIdx.x] = s;
     __syncthreads();
     for (int o = 128; o > 0; o >>= 1) {
          if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
          __syncthreads();
     }
     if (threadIdx.x == 0) mu[(size_t)b * nblk + j] = (T)(red[0] / (2. * 4096));
}

template <typename T>
__device__ __forceinline__ T fval(const T *Fb, const T *mub, int k, int fr0, int nblk) {
     T f = Fb[k];
     if (mub) {
          const int r = k - fr0;
          if (r < nblk * 4096) f = f / mub[r >> 12];
     }
     return f;
}

template <typename T>
__device__ __forceinline__ bool is_peak(const T *Fb, const T *mub, int k, int fr0, int nblk, double thr) {
     const T f = fval(Fb, mub, k, fr0, nblk);
     return !(f < thr || fval(Fb, mub, k - 1, fr0, nblk) > f || f < fval(Fb, mub, k + 1, fr0, nblk));
}

struct ThrArgs {
     int nF, fr0, fr1;
     double thr;
     int nblk;
     const TmplParam *tp;
     int nfftf;
     const double *lines;
     int numlines;
     unsigned bufhalf;
     Trig *trig;
     unsigned long long cap;
     unsigned long long *cnt;
     unsigned *tcnt;
     unsigned *err;
};

// Appends the trigger at bin i of template b (group-relative) with F value
// Fc: its frequency (jobcore.c:571) in the emulated build's arithmetic, the
// veto intervals (jobcore.c:575-583), the per-template count against
// bufsize/2 (jobcore.c:586-590), then the compacted trigger list.
template <bool FP64>
__device__ __forceinline__ void emit_trigger(const ThrArgs &A, int b, int i, double Fc)
{
     const TmplParam P = A.tp[b];
     double fcmp;
     float ff;
     if (FP64) {
          // FLOAT_TYPE = double: f_ = (double)(2ic)/(double)nfftf*M_PI + sgnl0
          const double f_ = __dadd_rn(__dmul_rn(__ddiv_rn((double)(2 * i), (double)A.nfftf), M_PI_D), P.sgnl0);
          fcmp = f_;
          ff = (float)f_;
     } else {
          // FLOAT_TYPE = float: the quotient in float, the product and sum in
          // double, stored to float
          const float qf = __fdiv_rn((float)(2 * i), (float)A.nfftf);
          ff = (float)__dadd_rn(__dmul_rn((double)qf, M_PI_D), P.sgnl0);
          fcmp = (double)ff;
     }
     for (int k = 0; k < A.numlines; k++)
          if (fcmp >= A.lines[2 * k] && fcmp <= A.lines[2 * k + 1]) return;
     const unsigned c = atomicAdd(&A.tcnt[b], 1u);
     if (c >= A.bufhalf) {
          atomicOr(A.err, ERR_OVERFLOW);
          return;
     }
     const unsigned long long g = atomicAdd(A.cnt, 1ull);
     if (g < A.cap) {
          Trig r;
          r.id = P.id;
          r.bin = (uint32_t)i;
          r.f = ff;
          r.F = (float)Fc;
          A.trig[g] = r;
     }
}

// MAX_ALG 3 (jobcore.c:556-603) as the single-threaded loop executes it:
// bin i (fr0 < i < fr1-1) is a trigger when it is a local maximum >= thr
// and the previous accepted bin is not i-1 (the loop's "i++" skip), i.e.
// when the run of consecutive local-maximum bins ending at i-1 has even
// length.  Then the veto intervals are checked and the trigger appended.
template <typename T, bool FP64>
__device__ __forceinline__ void threshold_bin(const T *__restrict__ F, const T *__restrict__ mu, const ThrArgs &A,
                                              int b, int i)
{
     const int fr0 = A.fr0, nblk = A.nblk;
     const double thr = A.thr;
     const T *Fb = F + (size_t)b * A.nF - fr0;
     const T *mub = mu ? mu + (size_t)b * nblk : nullptr;
     if (!is_peak(Fb, mub, i, fr0, nblk, thr)) return;
     int run = 0;
     for (int k = i - 1; k >= fr0 + 1 && is_peak(Fb, mub, k, fr0, nblk, thr); k--) run++;
     if (run & 1) return;
     emit_trigger<FP64>(A, b, i, (double)fval(Fb, mub, i, fr0, nblk));
}

// The candidates the row pass collected; when the list overflowed, every
// bin of the chunk (grid-stride).  grid (G), 256 threads
template <typename T, bool FP64>
__global__ void __launch_bounds__(256) k_resolve(const T *__restrict__ F, ThrArgs A, const uint2 *__restrict__ cand,
                                                 const unsigned *__restrict__ cand_cnt, unsigned cand_cap, int nt)
{
     const unsigned n = *cand_cnt;
     const unsigned gs = gridDim.x * blockDim.x;
     const unsigned g0 = blockIdx.x * blockDim.x + threadIdx.x;
     if (n <= cand_cap) {
          for (unsigned c = g0; c < n; c += gs) {
               const uint2 q = cand[c];
               threshold_bin<T, FP64>(F, nullptr, A, (int)q.x, (int)q.y);
          }
     } else {
          const unsigned nb = (unsigned)(A.fr1 - A.fr0 - 2 > 0 ? A.fr1 - A.fr0 - 2 : 0);   // bins fr0+1 .. fr1-2
          for (unsigned long long x = g0; x < (unsigned long long)nt * nb; x += gs)
               threshold_bin<T, FP64>(F, nullptr, A, (int)(x / nb), A.fr0 + 1 + (int)(x % nb));
     }
}

// Trigger selection from the sparse F store's candidate records: the
// missing neighbour of a run's end bin from the edge ring, the local-maximum
// test, and the trigger append.  A record whose MAX_ALG 3 run needs more of
// the spectrum (a tie with the previous bin), or a candidate list that
// overflowed, sets ERR_NEED_FULL_F: the host then reruns the batch with the
// full F store.  grid (G), 256 threads
struct SparseArgs {
     const float *E;
     const uint4 *cand;
     const unsigned *cand_cnt;
     unsigned cand_cap;
     int N1, L;       // four-step column count and row length
};

__global__ void __launch_bounds__(256) k_resolve_sparse(ThrArgs A, SparseArgs S)
{
     const unsigned n = *S.cand_cnt;
     if (n > S.cand_cap) {
          if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(A.err, ERR_NEED_FULL_F);
          return;
     }
     const unsigned gs = gridDim.x * blockDim.x;
     const int nj = S.N1 / RUN;
     for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gs) {
          const uint4 r = S.cand[i];
          const int b = (int)(r.x & 0xffffffu);
          const unsigned kind = r.x >> 24;
          const int k = (int)r.y;
          const float f = __uint_as_float(r.z);
          if (kind == CAND_TIE) {
               atomicOr(A.err, ERR_NEED_FULL_F);
               continue;
          }
          if (kind != CAND_LOCAL) {
               const int k1 = k % S.N1, k2 = k / S.N1, j = k1 / RUN;
               const float *Eb = S.E + (size_t)b * nj * (2 * S.L);
               float fm, fp;
               if (kind == CAND_LEFT) {
                    // bin k-1: the last bin of the previous CTA's run (or of the last CTA's at k2-1)
                    fm = j > 0 ? Eb[((size_t)(j - 1) * S.L + k2) * 2 + 1] : Eb[((size_t)(nj - 1) * S.L + (k2 - 1)) * 2 + 1];
                    fp = __uint_as_float(r.w);
               } else {
                    // bin k+1: the first bin of the next CTA's run (or of the first CTA's at k2+1)
                    fp = j < nj - 1 ? Eb[((size_t)(j + 1) * S.L + k2) * 2] : Eb[((size_t)k2 + 1) * 2];
                    fm = __uint_as_float(r.w);
               }
               if (fm > f || f < fp) continue;   // not a local maximum
               if (fm == f) {
                    atomicOr(A.err, ERR_NEED_FULL_F);
                    continue;
               }
          }
          emit_trigger<false>(A, b, k, (double)f);
     }
}

// Full scan of every bin (used with the blocks_avg normalisation).  A thread
// looks at 8 bins of one block, so that a CTA has one mean; bins clearly below
// the threshold are passed over by a product instead of the exact quotient
// (one bin per thread and a division each took 29 us for 64 templates of
// 127,000 bins, 12 us now).  grid (ceil(nF/2048), ntmpl), 256 threads
template <typename T, bool FP64>
__global__ void __launch_bounds__(256) k_threshold(const T *__restrict__ F, const T *__restrict__ mu, ThrArgs A)
{
     const int b = blockIdx.y, r0 = blockIdx.x * 2048 + threadIdx.x;
     const T *Fb = F + (size_t)b * A.nF;
     T lim = -CUDART_INF;
     if (A.thr > 0.) {
          const int j = (blockIdx.x * 2048) >> 12;
          lim = (T)(A.thr * (1. - 1e-5) * (mu && j < A.nblk ? (double)mu[(size_t)b * A.nblk + j] : 1.));
     }
     T v[8];
#pragma unroll
     for (int k = 0; k < 8; k++) v[k] = r0 + 256 * k < A.nF ? Fb[r0 + 256 * k] : lim;
#pragma unroll
     for (int k = 0; k < 8; k++) {
          const int i = A.fr0 + r0 + 256 * k;
          if (i < A.fr0 + 1 || i >= A.fr1 - 1 || v[k] < lim) continue;
          threshold_bin<T, FP64>(F, mu, A, b, i);
     }
}

}  // namespace tdf
