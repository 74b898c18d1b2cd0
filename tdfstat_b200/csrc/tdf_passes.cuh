// tdf_passes.cuh -- the two four-step pass kernels (see tdf_fft.cuh) and the
// prologue/epilogue policies fused into them.
//
//   k_colpass<T, L, SIGN, NA, Pro, Epi>: CTA = LINES columns n2 of an
//     N = L*N2 transform, L threads; Pro::load fills the first-pass inputs
//     x[N2*n1 + n2] straight into registers (coalesced across the 8 columns),
//     Epi::store consumes the outputs k1 = t + m*L/8.
//   k_rowpass<T, L, SIGN, NA, Src, Epi>: CTA = LINES rows k1 of an
//     N = N1*L transform, L threads; the first-pass inputs are loaded from
//     the rows straight into registers, Epi::store consumes X[k1 + N1*k2].
// They run the sky stage's transforms for interpolation factors other than two
// and the allocation-free FP32 entry point; the spindown passes of both forms
// are in tdf_split.cuh, the interpolation by two in tdf_sky.cuh.
#pragma once

#include <type_traits>

#include "tdf_fft.cuh"

namespace tdf {

// threads of a pass CTA: L/8 per line, LINES lines
template <int L>
constexpr int pass_threads() { return L / 8 * LINES; }

template <typename T, int L, int NA>
constexpr size_t pass_smem_bytes() {
     return sizeof(cx<T>) * (L + (size_t)NA * LINES * LineGeom<T, L>::STRIDE);
}

// resident CTAs per SM the passes are compiled for (register cap): FP32
// column passes and row passes; FP64 passes at 64 registers (two CTAs of 512
// threads fit the shared memory)
template <typename T, int L>
constexpr int pass_min_blocks() {
     return sizeof(T) == 4 ? (L <= 256 ? 3 : (L == 512 ? 2 : 1)) : (1024 / L > 1 ? 1024 / L : 1);
}
template <typename T, int L>
constexpr int row_min_blocks() {
     return sizeof(T) == 4 ? (L <= 256 ? 4 : (L == 512 ? 2 : 1)) : (1024 / L > 1 ? 1024 / L : 1);
}

// An epilogue with `static constexpr bool kTables = true` keeps tables in
// dynamic shared memory at byte offset tab_off: load_tables<L>() fills them
// before the first barrier and store() gets the shared memory base.
template <class P, class = void>
struct has_tables : std::false_type {};
template <class P>
struct has_tables<P, std::void_t<decltype(P::kTables)>> : std::integral_constant<bool, P::kTables> {};

// The column pass of CTA (blk, b): columns n2 = blk*LINES + c of batch b.
template <typename T, int L, int SIGN, int NA, class Pro, class Epi>
__device__ __forceinline__ void col_body(const Pro &pro, const Epi &epi, const cx<T> *__restrict__ twline, int blk,
                                         int b, unsigned char *smem_raw) {
     using G = LineGeom<T, L>;
     cx<T> *tw = reinterpret_cast<cx<T> *>(smem_raw);
     cx<T> *lines = tw + L;
     load_table<T>(tw, twline, L);
     if constexpr (has_tables<Epi>::value) epi.template load_tables<L>(smem_raw);
     const int tid = threadIdx.x;
     const int c = tid % LINES, t = tid / LINES;
     const int n2 = blk * LINES + c;
     cx<T> v[NA][8];
     pro.template load<L>(v, b, n2, t);
     cx<T> *s[NA];
#pragma unroll
     for (int a = 0; a < NA; a++) s[a] = lines + (a * LINES + c) * G::STRIDE;
     __syncthreads();
     line_fft<T, L, SIGN, NA>(v, s, tw, t);
     if constexpr (has_tables<Epi>::value)
          epi.template store<L>(v, b, n2, t, smem_raw);
     else
          epi.template store<L>(v, b, n2, t);
}

// The row pass of CTA (blk, b): rows k1 = blk*LINES + c of batch b.
template <typename T, int L, int SIGN, int NA, class Src, class Epi>
__device__ __forceinline__ void row_body(const Src &src, const Epi &epi, const cx<T> *__restrict__ twline, int blk,
                                         int b, unsigned char *smem_raw) {
     using G = LineGeom<T, L>;
     cx<T> *tw = reinterpret_cast<cx<T> *>(smem_raw);
     cx<T> *lines = tw + L;
     const int tid = threadIdx.x;
     const int k1b = blk * LINES;
     const int c = tid % LINES, t = tid / LINES;
     cx<T> v[NA][8];
     cx<T> *s[NA];
     // first-pass inputs straight from the rows into registers: per load
     // instruction a warp reads 4 consecutive elements of each of 8 rows
     src.template load<L>(v, b, k1b + c, t);
     load_table<T>(tw, twline, L);
#pragma unroll
     for (int a = 0; a < NA; a++) s[a] = lines + (a * LINES + c) * G::STRIDE;
     __syncthreads();
     line_fft<T, L, SIGN, NA>(v, s, tw, t);
     epi.template store<L>(v, b, k1b + c, t);
}

template <typename T, int L, int SIGN, int NA, class Pro, class Epi>
__global__ void __launch_bounds__(pass_threads<L>(), (pass_min_blocks<T, L>()))
k_colpass(const __grid_constant__ Pro pro, Epi epi, const cx<T> *__restrict__ twline) {
     extern __shared__ __align__(128) unsigned char smem_raw[];
     col_body<T, L, SIGN, NA>(pro, epi, twline, blockIdx.x, blockIdx.y, smem_raw);
}

template <typename T, int L, int SIGN, int NA, class Src, class Epi>
__global__ void __launch_bounds__(pass_threads<L>(), (row_min_blocks<T, L>())) k_rowpass(Src src, Epi epi, const cx<T> *__restrict__ twline) {
     extern __shared__ __align__(128) unsigned char smem_raw[];
     row_body<T, L, SIGN, NA>(src, epi, twline, blockIdx.x, blockIdx.y, smem_raw);
}

// ------------------------------------------------------------------ policies

// Column-pass epilogue: multiply by W_N^(n2*k1) and store Y[k1*N2 + n2].
// Batch b's arrays are interleaved element by element: array a of element e
// lives at y[((size_t)b*N + e)*NA + a], so both arrays of a sample move in one
// access (16 bytes for two float2).
// The twiddle tables hi[L*N2/1024] = W^(1024 i), lo[1024] = W^j are copied
// into dynamic shared memory at byte offset tab_off (set by the launcher) when
// the kernel starts, in the same batch of loads as the line table.  FP32
// passes form a thread's eight twiddles W^(n2 (t + m L/8)) by recurrence from
// W^(n2 t) and W^(n2 L/8) (relative error below 1e-6); FP64 passes look each
// one up.
template <typename T, int SIGN, int NA>
struct StoreFourstep {
     cx<T> *y;
     const cx<T> *hi, *lo;
     int N2;
     int N;                 // array stride
     unsigned tab_off = 0;  // byte offset of the shared copies of hi, lo
     static constexpr bool kTables = true;

     template <int L>
     __host__ __device__ static constexpr int nhi(int N2) { return L * N2 / 1024; }
     template <int L>
     __host__ __device__ static size_t table_bytes(int N2) { return sizeof(cx<T>) * (size_t)(nhi<L>(N2) + 1024); }

     template <int L>
     __device__ __forceinline__ void load_tables(unsigned char *smem) const {
          cx<T> *s = reinterpret_cast<cx<T> *>(smem + tab_off);
          const int nh = nhi<L>(N2);
          for (int i = threadIdx.x; i < nh + 1024; i += blockDim.x) s[i] = i < nh ? __ldg(&hi[i]) : __ldg(&lo[i - nh]);
     }

     template <int L>
     __device__ __forceinline__ void store(const cx<T> (&v)[NA][8], int b, int n2, int t, unsigned char *smem) const {
          const cx<T> *hs = reinterpret_cast<const cx<T> *>(smem + tab_off);
          const cx<T> *ls = hs + nhi<L>(N2);
          cx<T> w = twsign<SIGN>(fourstep_twiddle_smem<T>(hs, ls, n2 * t));
          cx<T> st = w;
          if constexpr (sizeof(T) == 4) st = twsign<SIGN>(fourstep_twiddle_smem<T>(hs, ls, n2 * (L / 8)));
#pragma unroll
          for (int m = 0; m < 8; m++) {
               const int k1 = t + m * (L / 8);
               if constexpr (sizeof(T) == 4) {
                    if (m > 0) w = cmul(w, st);
               } else {
                    w = twsign<SIGN>(fourstep_twiddle_smem<T>(hs, ls, n2 * k1));
               }
               cx<T> *dst = y + ((size_t)b * N + n2 + (size_t)k1 * N2) * NA;
               if constexpr (NA == 2 && sizeof(T) == 4) {
                    const cx<T> p = cmul(v[0][m], w), q = cmul(v[1][m], w);
                    *reinterpret_cast<float4 *>(dst) = make_float4(p.x, p.y, q.x, q.y);
               } else {
#pragma unroll
                    for (int a = 0; a < NA; a++) dst[a] = cmul(v[a][m], w);
               }
          }
     }
};

// Row-pass source: rows of Y laid out as in StoreFourstep.  load() fills the
// first-pass inputs v[a][m] = row k1 element t + m*L/8 of every array.
template <typename T, int NA>
struct RowsY {
     const cx<T> *y;
     int N;          // N1*N2
     int rowstride;  // N2
     template <int L>
     __device__ __forceinline__ void load(cx<T> (&v)[NA][8], int b, int k1, int t) const {
          const cx<T> *r = y + ((size_t)b * N + (size_t)k1 * rowstride) * NA;
#pragma unroll
          for (int m = 0; m < 8; m++) {
               const cx<T> *e = r + (size_t)(t + m * (L / 8)) * NA;
               if constexpr (NA == 2 && sizeof(T) == 4) {
                    const float4 q = *reinterpret_cast<const float4 *>(e);
                    v[0][m] = make_float2(q.x, q.y);
                    v[1][m] = make_float2(q.z, q.w);
               } else {
#pragma unroll
                    for (int a = 0; a < NA; a++) v[a][m] = e[a];
               }
          }
     }
};

// Row-pass epilogue: natural-order output X[k1 + N1*k2] for k < nkeep and
// k = klast.
template <typename T>
struct StoreNatural {
     cx<T> *x;
     int N1;
     int N;          // array stride
     int nkeep, klast;
     template <int L>
     __device__ __forceinline__ void store(const cx<T> (&v)[1][8], int b, int k1, int t) const {
          cx<T> *dst = x + (size_t)b * N;
#pragma unroll
          for (int m = 0; m < 8; m++) {
               int k = k1 + N1 * (t + m * (L / 8));
               if (k < nkeep || k == klast) dst[k] = v[0][m];
          }
     }
};

// The same with arrays 2q and 2q + 1 interleaved: element k of the pair q is
// (re, re, im, im) at x[(q*N + k)*4].
struct StorePairs {
     double *x;
     int N1;
     int N;
     int nkeep, klast;
     template <int L>
     __device__ __forceinline__ void store(const double2 (&v)[1][8], int b, int k1, int t) const {
          double *dst = x + (size_t)(b >> 1) * N * 4 + (b & 1);
#pragma unroll
          for (int m = 0; m < 8; m++) {
               const int k = k1 + N1 * (t + m * (L / 8));
               if (k < nkeep || k == klast) {
                    dst[(size_t)k * 4] = v[0][m].x;
                    dst[(size_t)k * 4 + 2] = v[0][m].y;
               }
          }
     }
};

// Column-pass prologue: plain load of x[N2*n1 + n2] from natural-order arrays
// of stride N (arrays already zero-padded to N).
template <typename T>
struct LoadNatural {
     const cx<T> *x;
     int N2;
     int N;
     template <int L>
     __device__ __forceinline__ void load(cx<T> (&v)[1][8], int b, int n2, int t) const {
          const cx<T> *src = x + (size_t)b * N + n2;
#pragma unroll
          for (int m = 0; m < 8; m++) v[0][m] = src[(size_t)N2 * (t + m * (L / 8))];
     }
};

// Column-pass prologue of the interpolation inverse FFT: the spectrum of
// length nfft is spread to Ninterp = ratio*nfft, moving bins [nyqst, nfft)
// to the top and zeroing the middle (jobcore.c:336-350), and multiplied by
// fac (k_interp_factor).
template <typename T>
struct LoadShuffled {
     const cx<T> *x;  // forward spectra (nfft values each), arrays `stride` apart
     const T *fac;
     int N2;          // of the Ninterp transform
     int stride;
     int nfft;
     int Ninterp;
     template <int L>
     __device__ __forceinline__ void load(cx<T> (&v)[1][8], int b, int n2, int t) const {
          const cx<T> *src = x + (size_t)b * stride;
          const int nyqst = nfft / 2 + 1;
          const int gap = Ninterp - nfft;
#pragma unroll
          for (int m = 0; m < 8; m++) {
               int k = N2 * (t + m * (L / 8)) + n2;
               cx<T> z;
               z.x = 0;
               z.y = 0;
               if (k < nyqst) z = cscale(src[k], fac[k]);
               else if (k >= nyqst + gap) z = cscale(src[k - gap], fac[Ninterp - k]);
               v[0][m] = z;
          }
     }
};

// fac[k] = scale * 6/(4 + 2 cos(2 pi k/Ninterp)), k <= nfft/2: the scale of
// the inverse interpolation FFT and the frequency response of the cubic
// B-spline prefilter, so that the transform yields the spline coefficients c
// of the interpolated series y, y[k] = (c[k-1] + 4 c[k] + c[k+1])/6 (periodic;
// the natural end conditions are put in by splint_eval).
__global__ void k_interp_factor(double *fac, int n, double dw, double scale) {
     const int k = blockIdx.x * blockDim.x + threadIdx.x;
     if (k < n) fac[k] = scale * 6. / (4. + 2. * cospi(dw * k));
}

}  // namespace tdf
