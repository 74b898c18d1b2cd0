// tdf_sky.cuh -- the sky stage (FP64, once per sky point and detector;
// jobcore.c:283-391): modulation and time shift, interpolation by FFT to twice
// the rate, spline resampling.  Four kernels:
//
//   k_sky_col    modvir + barycentric shift + phase modulation of a column's
//                samples (settings.c:254-294, jobcore.c:283-312), the first
//                pass of the forward FFT; partial sums of aa^2, bb^2
//   k_sky_mid    the rows of the forward FFT and the columns of the inverse one
//   k_row        (CoefRow) the rows of the inverse FFT, which leave the spline
//                coefficients of the interpolated series
//   k_splint     natural-spline evaluation at 2(i - shftf[i]) (auxi.c:93-169),
//                division by sig2, conversion to the spindown operands; aa, bb
//                network sums (FLOAT_TYPE emulation per form)
//
// The two arrays (a, b) of a point and detector are transformed as one pair,
// with the thread groups, exchanges and block layouts of the FP64 spindown
// passes (tdf_split.cuh): 66 us per point of six days and two detectors in
// batches of eight (86 with separate arrays, CTA-wide barriers and the
// modulation in a kernel of its own).
// The inverse transform runs as a forward one on values whose real and
// imaginary parts are swapped.
//
// With another interpolation factor than two the FFT passes run apart
// (k_sky_prep, then tdf_passes.cuh).
#pragma once

namespace tdf {

// shft_n[i] = n . DetSSB[i], without FMA contraction: the phase made from it
// reaches ~1e5 rad, so its rounding must follow the reference's
__device__ __forceinline__ double shft_of(const SkyParam &S, double e0, double e1, double e2) {
     return __dadd_rn(__dadd_rn(__dmul_rn(S.nS0, e0), __dmul_rn(S.nS1, e1)), __dmul_rn(S.nS2, e2));
}
__device__ __forceinline__ double shft_at(const SkyParam &S, const double *e) {
     return shft_of(S, __ldg(e), __ldg(e + 1), __ldg(e + 2));
}

// what a sample's modulation reads
struct SkySample {
     float x;
     double cosm, sinm, e0, e1, e2;
};

// sample i of the modulated pair: x (aa, bb) e^{-i (het0 i + oms shft)}; aa^2
// and bb^2 are added to a2 and b2.  LIB: the library's sine and cosine (phases
// past 2^30 rad); `far` collects the largest phase.
template <bool LIB>
__device__ __forceinline__ D2 sky_sample(const SkyParam &S, const DetParam &D, const SkySample &q, int i, double oms,
                                         double &a2, double &b2, double &far) {
     double aa, bb;
     modvir_at(D, S.sinalt, S.cosalt, S.sindelt, S.cosdelt, q.cosm, q.sinm, q.x, aa, bb);
     const double phase = __dadd_rn(__dmul_rn(S.het0, (double)i), __dmul_rn(oms, shft_of(S, q.e0, q.e1, q.e2)));
     far = fmax(far, fabs(phase));
     double sn, cn;
     if (LIB) sincos_large(phase, &sn, &cn);
     else sincos_spin(phase, sn, cn);
     const double ra = (double)q.x * aa, rb = (double)q.x * bb;
     a2 += aa * aa;
     b2 += bb * bb;
     return D2{make_double2(ra * cn, rb * cn), make_double2(ra * -sn, rb * -sn)};
}

struct SkyCol {
     const float *xdat;
     const double *detssb, *cosm, *sinm;
     const SkyParam *sp;
     const DetParam *dp;
     int nifo, N, Nal, N2;
     double oms;
     double2 *y;
     const double2 *w0, *ws, *ltw;   // as in Fp64Col, of the nfft transform
     double *partial;                // [q][N2/lines*warps][2]
};

// twiddle W^(n2 k1) of output m and the store of a column's value into its
// block of four k1 (k1 = t + m L/8 of column n2; blocks of N2 columns)
template <int L>
__device__ __forceinline__ void store_col64(D2 (&v)[8], double2 *y, const double2 *__restrict__ w0,
                                            const double2 *__restrict__ ws, int N2, int n2, int t) {
     constexpr int R = run_of<double2>;
     const double2 w = __ldg(&w0[n2 * (L / 8) + t]);
     double2 *dst = y + (size_t)(t / R) * (2 * R * N2) + n2 * R + t % R;
#pragma unroll
     for (int m = 0; m < 8; m++) {
          const D2 q = pcmul(v[m], m == 0 ? w : cmul_tw(w, __ldg(&ws[n2 * 8 + m])));
          double2 *d = dst + (size_t)m * (L / 8 / R) * (2 * R * N2);
          d[0] = q.re;
          d[R * N2] = q.im;
     }
}

// The lanes of a warp are four columns at eight rows: the samples come in
// natural order, so a load touches eight rows' lines of 128 bytes.  With the 32
// rows of one column per warp it touched 32 (L1 49% busy on them, the load
// queue full): 75 -> 66 us per sky point of 2^18 samples for the whole stage,
// 31.2 -> 28.5 for 2^17, 15.0 -> 13.9 for 2^16 (two detectors, batches).
// grid (N2 / fp64_col_lines<L>(), Q)
template <int L>
__global__ void __launch_bounds__(fp64_col_threads<L>(), 512 / fp64_col_threads<L>())
k_sky_col(const __grid_constant__ SkyCol a) {
     extern __shared__ __align__(128) unsigned char smem_raw[];
     using G = SplitLine<double2, L, true>;
     constexpr int R = run_of<double2>;
     const int grp = threadIdx.x / (L / 2), c = threadIdx.x % R, t = threadIdx.x % (L / 2) / R;
     const int n2 = blockIdx.x * fp64_col_lines<L>() + grp * R + c, q = blockIdx.y, d = q % a.nifo;
     const SkyParam S = a.sp[q / a.nifo];
     const DetParam &D = a.dp[d];
     D2 v[1][8];
     double s2 = 0., t2 = 0., far = 0.;
     // straight-line code, a sample's inputs loaded one ahead; samples past the
     // end read the last one's with x = 0 and give zeros
     auto load = [&](int m) {
          const int i = a.N2 * (t + m * (L / 8)) + n2, j = min(i, a.N - 1);
          const double *e = a.detssb + ((size_t)d * a.N + j) * 3;
          SkySample q{ldg1_v(&a.xdat[(size_t)d * a.Nal + j]), ldgd_v(&a.cosm[j]), ldgd_v(&a.sinm[j]),
                      ldgd_v(e), ldgd_v(e + 1), ldgd_v(e + 2)};
          if (i >= a.N) q.x = 0.f;
          return q;
     };
     SkySample cur = load(0);
#pragma unroll
     for (int m = 0; m < 8; m++) {
          SkySample nxt;
          if (m < 7) nxt = load(m + 1);
          v[0][m] = sky_sample<false>(S, D, cur, a.N2 * (t + m * (L / 8)) + n2, a.oms, s2, t2, far);
          if (m < 7) cur = nxt;
     }
     if (!(far < 1073741824.)) {
          s2 = t2 = 0.;
#pragma unroll
          for (int m = 0; m < 8; m++)
               v[0][m] = sky_sample<true>(S, D, load(m), a.N2 * (t + m * (L / 8)) + n2, a.oms, s2, t2, far);
     }
#pragma unroll
     for (int o = 16; o > 0; o >>= 1) {
          s2 += __shfl_down_sync(0xffffffffu, s2, o);
          t2 += __shfl_down_sync(0xffffffffu, t2, o);
     }
     if (threadIdx.x % 32 == 0) {
          constexpr int W = fp64_col_threads<L>() / 32;
          double *p = a.partial + (((size_t)q * gridDim.x + blockIdx.x) * W + threadIdx.x / 32) * 2;
          p[0] = s2;
          p[1] = t2;
     }
     split_fft<L, true, 1>(v, smem_raw + grp * G::BYTES + c * (G::STRIDE * sizeof(double2)), 0, a.ltw, t, grp, [] {});
     store_col64<L>(v[0], a.y + (size_t)q * (2 * L * a.N2), a.w0, a.ws, a.N2, n2, t);
}

// Forward rows and inverse columns when Ninterp = 2 nfft.  With nfft = N1*L
// (rows of L points) the inverse transform has N1 columns of 2L points, and
// the outputs X[k1 + N1*k2] of forward row k1 are exactly the inputs of inverse
// column k1, so the spectrum never goes to memory.  Half of an inverse
// column's inputs are the zero padding (jobcore.c:336-350), the others are
// multiplied by fac (k_interp_factor).
struct SkyMid {
     const double2 *y;
     double2 *z;
     const double2 *ltw1;            // pass twiddles of L and of 2L points
     const double2 *ltw2;
     const double2 *w0, *ws;         // of the Ninterp transform
     const double *fac;
     int N1;
};

// One CTA: a block of four rows, L threads; the forward rows use half of them.
// grid (N1/4, Q)
template <int L>
__global__ void __launch_bounds__(L, 512 / L) k_sky_mid(const __grid_constant__ SkyMid a) {
     extern __shared__ __align__(128) unsigned char smem_raw[];
     constexpr int R = run_of<double2>;
     using G1 = SplitLine<double2, L, true>;
     using G2 = SplitLine<double2, 2 * L, true>;
     const int c = threadIdx.x % R, t = threadIdx.x / R;
     const int k1 = blockIdx.x * R + c, q = blockIdx.y;
     const bool fwd = t < L / 8;
     D2 v[1][8];
     if (fwd) {
          const double2 *src = a.y + ((size_t)q * (a.N1 / R) + blockIdx.x) * (2 * R * L) + threadIdx.x;
#pragma unroll
          for (int m = 0; m < 8; m++) v[0][m] = D2{__ldg(src + m * (L / 8 * R)), __ldg(src + L * R + m * (L / 8 * R))};
     }
     split_fft<L, true, 1, L>(v, smem_raw + c * (G1::STRIDE * sizeof(double2)), 0, a.ltw1, t, 0, [] {}, fwd);
     __syncthreads();   // the last exchange is read
     unsigned char *s = smem_raw + c * (G2::STRIDE * sizeof(double2));
     if (fwd) {
          const int nfft = a.N1 * L;
#pragma unroll
          for (int m = 0; m < 8; m++) {
               const int k2 = t + m * (L / 8), k = k1 + a.N1 * k2;
               const double2 f = pdup(__ldg(&a.fac[k <= nfft / 2 ? k : nfft - k]));
               // real and imaginary parts swapped from here on
               G2::put(s, G2::pos(k2), D2{pmul(v[0][m].im, f), pmul(v[0][m].re, f)});
          }
     }
     __syncthreads();
     // input n1 = t + m L/4 of the inverse column: bins k2 = n1 below nfft/2,
     // k2 = n1 - L in the top quarter; bin nfft/2 itself (row 0) on the low side
#pragma unroll
     for (int m = 0; m < 8; m++) {
          const int n1 = t + m * (L / 4);
          v[0][m] = m < 2 ? G2::get(s, G2::pos(n1)) : (m >= 6 ? G2::get(s, G2::pos(n1 - L)) : pzero_of<double2>());
     }
     if (k1 == 0 && t == 0) {
          v[0][2] = v[0][6];
          v[0][6] = pzero_of<double2>();
     }
     __syncthreads();
     split_fft<2 * L, true, 1, L>(v, s, 0, a.ltw2, t, 0, [] {});
     store_col64<2 * L>(v[0], a.z + (size_t)q * (4 * L * a.N1), a.w0, a.ws, a.N1, k1, t);
}

// The rows of the inverse transform: coefficients c[k], k = k1 + N1*k2, of pair
// b for k < nkeep and k = klast.
struct CoefRow {
     using V = double2;
     const double2 *y;
     const double2 *ltw;
     D2 *c;
     size_t stride;
     int nkeep, klast;
     int nt;          // pairs
     unsigned *err;
     int probes;      // limit of the waits for a row block
};

template <int L, int N1, bool HALF, class F>
__device__ __forceinline__ void split_row_block(const CoefRow &a, int b, int blk, int tid, int id, const double2 *y, bool,
                                                unsigned char *lines, const F &read) {
     constexpr int R = run_of<double2>;
     const int c = tid % R, t = tid / R;
     D2 v[1][8];
#pragma unroll
     for (int m = 0; m < 8; m++) {
          v[0][m].re = y[tid + m * (L / 8 * R)];
          v[0][m].im = y[L * R + tid + m * (L / 8 * R)];
     }
     group_sync<L / 2>(id);   // the exchanges reuse the rows' memory
     split_fft<L, true, 1>(v, lines + c * (SplitLine<double2, L, true>::STRIDE * sizeof(double2)), 0, a.ltw, t, id, read);
     D2 *dst = a.c + (size_t)b * a.stride;
#pragma unroll
     for (int m = 0; m < 8; m++) {
          const int k = blk * R + c + N1 * (t + m * (L / 8));
          if (k < a.nkeep || k == a.klast) dst[k] = D2{v[0][m].im, v[0][m].re};   // swapped back
     }
}

// ------------------------------------------------------------------ other interpolation factors

// grid (ceil(nfft/256), Q = npts*nifo), 256 threads
__global__ void __launch_bounds__(256) k_sky_prep(
     const float *__restrict__ xdat, const double *__restrict__ detssb,
     const double *__restrict__ cosm, const double *__restrict__ sinm,
     const SkyParam *__restrict__ sp, const DetParam *__restrict__ dp,
     int nifo, int N, int nfft, int Nal, double oms,
     double2 *__restrict__ W, size_t Wstride, double *__restrict__ partial)
{
     const int q = blockIdx.y, p = q / nifo, d = q % nifo;
     const int i = blockIdx.x * 256 + threadIdx.x;
     double a2 = 0., b2 = 0.;
     if (i < nfft) {
          double2 xa = make_double2(0., 0.), xb = make_double2(0., 0.);
          if (i < N) {
               const double *e = detssb + ((size_t)d * N + i) * 3;
               const SkySample in{xdat[(size_t)d * Nal + i], cosm[i], sinm[i], e[0], e[1], e[2]};
               double far = 0.;
               const D2 v = sky_sample<true>(sp[p], dp[d], in, i, oms, a2, b2, far);
               xa = make_double2(v.re.x, v.im.x);
               xb = make_double2(v.re.y, v.im.y);
          }
          W[((size_t)q * 2 + 0) * Wstride + i] = xa;
          W[((size_t)q * 2 + 1) * Wstride + i] = xb;
     }
     // block partial sums of aa^2, bb^2
     __shared__ double ra_[8], rb_[8];
#pragma unroll
     for (int o = 16; o > 0; o >>= 1) {
          a2 += __shfl_down_sync(0xffffffffu, a2, o);
          b2 += __shfl_down_sync(0xffffffffu, b2, o);
     }
     const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
     if (l == 0) { ra_[w] = a2; rb_[w] = b2; }
     __syncthreads();
     if (threadIdx.x == 0) {
          double sa = 0., sb = 0.;
          for (int k = 0; k < 8; k++) { sa += ra_[k]; sb += rb_[k]; }
          partial[((size_t)q * gridDim.x + blockIdx.x) * 2 + 0] = sa;
          partial[((size_t)q * gridDim.x + blockIdx.x) * 2 + 1] = sb;
     }
}

// ------------------------------------------------------------------ resampling

// aa = sum_n sum_i aa_n^2/sig2_n (jobcore.c:373-386) of sky point p by one CTA
// of 256 threads; each detector's partials reduced by a fixed tree
// (reproducible), then accumulated over detectors into FLOAT_TYPE as the
// reference build does.
__device__ void sky_sums(const double *__restrict__ partial, int nblk, const DetParam *__restrict__ dp, int nifo, int p,
                         AaBb *__restrict__ out)
{
     __shared__ double ra[256], rb[256];
     double aa = 0., bb = 0.;
     float aaf = 0.f, bbf = 0.f;
     for (int d = 0; d < nifo; d++) {
          const double *pp = partial + (size_t)(p * nifo + d) * nblk * 2;
          double sa = 0., sb = 0.;
          for (int k = threadIdx.x; k < nblk; k += 256) { sa += pp[2 * k]; sb += pp[2 * k + 1]; }
          ra[threadIdx.x] = sa;
          rb[threadIdx.x] = sb;
          __syncthreads();
          for (int o = 128; o > 0; o >>= 1) {
               if (threadIdx.x < o) {
                    ra[threadIdx.x] += ra[threadIdx.x + o];
                    rb[threadIdx.x] += rb[threadIdx.x + o];
               }
               __syncthreads();
          }
          sa = ra[0];
          sb = rb[0];
          __syncthreads();
          aa += sa / dp[d].sig2;
          bb += sb / dp[d].sig2;
          aaf = (float)((double)aaf + sa / dp[d].sig2);
          bbf = (float)((double)bbf + sb / dp[d].sig2);
     }
     if (threadIdx.x == 0) {
          out[p].aa = aa;
          out[p].bb = bb;
          out[p].aaf = aaf;
          out[p].bbf = bbf;
     }
}

// The natural cubic spline (auxi.c:93-169) through y[0..n-1], evaluated at x
// from B-spline coefficients: with t = x - k, k = floor(x),
//   s(x) = sum_j w_j(t) c[k + j], j = -1..2 (the four cubic B-spline weights).
// c0 holds the coefficients of the periodic spline of the whole interpolated
// series (period np, a power of two), which the inverse FFT delivers; its
// second derivatives at the ends of the data, D0 and Dn, are not zero.  The
// natural spline has c[k] = c0[k] + a z^k + b z^(n-1-k), z = sqrt(3) - 2: both
// added terms leave every y[k] as it is (z + 4 + 1/z = 0) and change the
// second derivative by -6 times themselves, so
//   a + b z^(n-1) = D0/6,  a z^(n-1) + b = Dn/6.
// They decay by 0.27 per sample and are left out 64 samples from the ends
// (1e-37).  Replaces two recurrence sweeps over every series (u, y2): half of
// the sky stage's passes over memory.
__device__ __forceinline__ double zpow(int e) {
     constexpr double z = -0.26794919243112270647, iz = -3.7320508075688772935;
     if (e > 128) return 0.;   // below 1e-73
     double p = 1.;
     for (int i = 0; i < e; i++) p *= z;
     for (int i = 0; i > e; i--) p *= iz;
     return p;
}

// both arrays' spline at x; c0[k]: element k of the pair
__device__ __forceinline__ D2 splint_eval(const D2 *__restrict__ c0, int n, int np, double x)
{
     if (x < 0 || x > n - 1) return pzero_of<double2>();
     const int k = (int)floor(x);
     const double t = x - k, u = 1. - t;
     const double2 wm = pdup(u * u * u * (1. / 6.)), wd = pdup(t * t * t * (1. / 6.));
     const double2 wa = pdup((2. / 3.) - t * t * (1. - .5 * t)), wb = pdup((2. / 3.) - u * u * (1. - .5 * u));
     auto at = [&](int j) {
          const double2 *p = reinterpret_cast<const double2 *>(c0 + (j & (np - 1)));
          return D2{__ldg(p), __ldg(p + 1)};
     };
     const D2 cm = at(k - 1), ca = at(k), cb = at(k + 1), cd = at(k + 2);
     D2 r{pfma(wm, cm.re, pfma(wa, ca.re, pfma(wb, cb.re, pmul(wd, cd.re)))),
          pfma(wm, cm.im, pfma(wa, ca.im, pfma(wb, cb.im, pmul(wd, cd.im))))};
     if (k < 64 || k > n - 66) {
          constexpr double z = -0.26794919243112270647;
          const double2 sx = pdup(1. / 6.), m2 = pdup(-2.);
          auto bend = [&](int j) {   // second difference at j, over 6
               const D2 a = at(j - 1), b = at(j), c = at(j + 1);
               return D2{pmul(sx, padd(pfma(m2, b.re, a.re), c.re)), pmul(sx, padd(pfma(m2, b.im, a.im), c.im))};
          };
          const D2 D0 = bend(0), Dn = bend(n - 1);
          const double w = zpow(n - 1), q = 1. / (1. - w * w);
          const double ga = zpow(k - 1) * (wm.x + z * (wa.x + z * (wb.x + z * wd.x))) * q;        // of a
          const double gb = zpow(n - 3 - k) * (wd.x + z * (wb.x + z * (wa.x + z * wm.x))) * q;    // of b
          const double2 f0 = pdup(ga - gb * w), fn = pdup(gb - ga * w);
          r.re = pfma(f0, D0.re, pfma(fn, Dn.re, r.re));
          r.im = pfma(f0, D0.im, pfma(fn, Dn.im, r.im));
     }
     return r;
}

// The inputs of the resampling (jobcore.c:314-370): spline coefficients C of
// pair q = point*nifo + det, `stride` apart; and the sums' partials (the CTA
// of a point's first tile forms its aa and bb).
struct SplintIn {
     const D2 *C;
     size_t stride;
     const SkyParam *sp;
     const double *detssb;
     const DetParam *dp;
     int N, n, np, interpftpad, nifo;
     const double *partial;
     int nblk;
     AaBb *ab;
};

struct D4 {
     double x, y, z, w;
};

// Operands in the column layout of tdf_split.cuh: with i = N2*n1 + n2, split
// form (SPLIT)
//   xab[(q*N2 + n2)*CL + n1] = (a.re, b.re, a.im, b.im) in FP32
//   s2[((p*N2 + n2)*CL + n1)*nifo + d] = 2 i shft[i]
// FP64 form
//   xre, xim[(q*N2 + n2)*CL + n1] = (a.re, b.re), (a.im, b.im)
//   t1[(q*N2 + n2)*CL + n1] = i^2 + 2 i shft[i]
// A CTA takes a tile of 32 columns and 8 rows: it reads along i (32
// consecutive samples per warp) and, through shared memory, writes 8
// consecutive n1 of a column (128 bytes) at a time.
// grid (N2/32, ceil(ceil(N/N2)/8), Q), 256 threads
template <bool SPLIT>
__global__ void __launch_bounds__(256) k_splint(const __grid_constant__ SplintIn I, int N2, int CL,
                                                float4 *__restrict__ xab, float *__restrict__ s2out,
                                                double2 *__restrict__ xre, double2 *__restrict__ xim,
                                                double *__restrict__ t1)
{
     using X = typename std::conditional<SPLIT, float4, D4>::type;
     using S = typename std::conditional<SPLIT, float, double>::type;
     __shared__ X xs[32][9];
     __shared__ S ss[32][9];
     const int q = blockIdx.z, p = q / I.nifo, d = q % I.nifo;
     {
          const int c = threadIdx.x % 32, r = threadIdx.x / 32;
          const int i = N2 * (blockIdx.y * 8 + r) + blockIdx.x * 32 + c;
          if (i < I.N) {
               // xDatm{a,b}[i] = splint(interpftpad*(i - (shft[i] - shft[0])))/sig2
               const double *e = I.detssb + (size_t)d * 3 * I.N;
               const double sh = shft_at(I.sp[p], e + 3 * (size_t)i), sig2 = I.dp[d].sig2;
               const D2 y = splint_eval(I.C + (size_t)q * I.stride, I.n, I.np,
                                        I.interpftpad * (i - __dsub_rn(sh, shft_at(I.sp[p], e))));
               X v;
               v.x = y.re.x / sig2;
               v.y = y.re.y / sig2;
               v.z = y.im.x / sig2;
               v.w = y.im.y / sig2;
               xs[c][r] = v;
               const double di = (double)i, h = __dmul_rn((double)(2 * i), sh);
               ss[c][r] = SPLIT ? (S)(float)h : (S)__dadd_rn(__dmul_rn(di, di), h);
          }
     }
     __syncthreads();
     const int c = threadIdx.x / 8, r = threadIdx.x % 8;
     const int n1 = blockIdx.y * 8 + r, n2 = blockIdx.x * 32 + c;
     if (N2 * n1 + n2 < I.N) {
          const size_t o = ((size_t)q * N2 + n2) * CL + n1;
          const X v = xs[c][r];
          if constexpr (SPLIT) {
               xab[o] = v;
               s2out[(((size_t)p * N2 + n2) * CL + n1) * I.nifo + d] = ss[c][r];
          } else {
               xre[o] = make_double2(v.x, v.y);
               xim[o] = make_double2(v.z, v.w);
               t1[o] = ss[c][r];
          }
     }
     // the network sums of the point
     if (blockIdx.x == 0 && blockIdx.y == 0 && d == 0) sky_sums(I.partial, I.nblk, I.dp, I.nifo, p, I.ab);
}

}  // namespace tdf
