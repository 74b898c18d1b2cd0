// tdf_split.cuh -- the spindown passes of both forms (two arrays):
//
//   k_split_col /
//   k_fp64_col    demodulation of a template's samples, the N1-point FFTs of
//                 its columns and the four-step twiddle -> Y
//   k_row         the N2-point FFTs of the rows of Y and the F-statistic
//   k_spinpass    split form: both as one ordered launch of persistent CTAs
//                 (opt-in)
//
// V = float2 (split form) or double2 (FP64 form) is a pair of one component
// of both arrays.
//
// Arithmetic.  The two arrays (a, b) go through the same transform with the
// same twiddles, so every value is held as a P2: the real parts of both
// arrays in one pair of registers and the imaginary parts in another, and
// each operation is one packed FP32 instruction (add/mul/fma .f32x2).  The
// FP32 pipe does the same work (64 pairs per clock and SM, as 128 scalars),
// but in half the issue slots, which the passes' loads, shared-memory
// exchanges and address arithmetic share.
//
// Work per thread group.  A column is transformed by L/8 threads of its own,
// with a barrier of just those threads (none across a warp for L <= 256):
// CTA-wide barriers keep all warps in phase, computing together and waiting
// together, while columns of their own drift apart and one column's loads
// overlap another's butterflies.  That needs a column's data to be contiguous:
//   operands  xab[(slot*nifo + d)*N2 + n2][n1] float4 (a.re, b.re, a.im, b.im)
//             s2[slot*N2 + n2][n1][d]           (rows of CL >= N/N2 entries)
//   Y         [template][k1/RUN][n2][k1%RUN]  float4, likewise (re, im)
// (FP64: xre, xim double2 and t1 double in the same order of columns, Y in
// blocks of a real plane [n2][k1%RUN] double2 and an imaginary one).  The
// column pass reads 512 consecutive bytes per warp and load and writes Y in
// runs of RUN consecutive k1 (128-byte lines; FP64 64 bytes in each plane);
// the row pass reads one contiguous block per k1/RUN.
#pragma once

namespace tdf {

// consecutive k1 of Y = rows per row block, the run of consecutive bins it
// holds; a block has 128 N2 bytes in both forms
template <class V> constexpr int run_of = sizeof(V) == 8 ? 8 : 4;
constexpr int RUN = run_of<float2>;

// ------------------------------------------------------------------ packed arithmetic

// Scalar operations of the phases, not contracted; on the host they give the
// same bits (for tests there).
__host__ __device__ __forceinline__ int low_word(double x) {
#ifdef __CUDA_ARCH__
     return __double2loint(x);
#else
     long long q;
     memcpy(&q, &x, sizeof(q));
     return (int)q;
#endif
}
__host__ __device__ __forceinline__ float float_of_bits(unsigned q) {
#ifdef __CUDA_ARCH__
     return __uint_as_float(q);
#else
     float x;
     memcpy(&x, &q, sizeof(x));
     return x;
#endif
}
__host__ __device__ __forceinline__ double dadd(double a, double b) {
#ifdef __CUDA_ARCH__
     return __dadd_rn(a, b);
#else
     return a + b;
#endif
}
__host__ __device__ __forceinline__ double dsub(double a, double b) { return dadd(a, -b); }

__device__ __forceinline__ float2 padd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 pmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 pfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 psub(float2 a, float2 b) {
     float2 r;
     asm("{\n\t.reg .b64 x, y, z;\n\t"
         "mov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
         "sub.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
         : "=f"(r.x), "=f"(r.y)
         : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
     return r;
}
__device__ __forceinline__ float2 pdup(float x) { return make_float2(x, x); }
__device__ __forceinline__ double2 padd(double2 a, double2 b) { return make_double2(__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y)); }
__device__ __forceinline__ double2 psub(double2 a, double2 b) { return make_double2(__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y)); }
__device__ __forceinline__ double2 pmul(double2 a, double2 b) { return make_double2(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)); }
__device__ __forceinline__ double2 pfma(double2 a, double2 b, double2 c) { return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y)); }
__device__ __forceinline__ double2 pdup(double x) { return make_double2(x, x); }

// one complex value of both arrays: re = (a.re, b.re), im = (a.im, b.im)
template <class V> struct PV {
     V re, im;
};
using P2 = PV<float2>;
using D2 = PV<double2>;
template <class V> __device__ __forceinline__ PV<V> operator+(PV<V> a, PV<V> b) { return PV<V>{padd(a.re, b.re), padd(a.im, b.im)}; }
template <class V> __device__ __forceinline__ PV<V> operator-(PV<V> a, PV<V> b) { return PV<V>{psub(a.re, b.re), psub(a.im, b.im)}; }
template <class V> __device__ __forceinline__ PV<V> pzero_of() { return PV<V>{pdup(decltype(V::x)(0)), pdup(decltype(V::x)(0))}; }
__device__ __forceinline__ P2 pzero() { return pzero_of<float2>(); }
__device__ __forceinline__ float4 pack4(P2 a) { return make_float4(a.re.x, a.re.y, a.im.x, a.im.y); }
__device__ __forceinline__ P2 unpack4(float4 q) { return P2{make_float2(q.x, q.y), make_float2(q.z, q.w)}; }
// product of two twiddles; the rounding is fixed here, whatever the compiler
// would contract, so that every variant of a pass gives the same bits
__device__ __forceinline__ float2 cmul_tw(float2 a, float2 b) {
     return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)), __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ double2 cmul_tw(double2 a, double2 b) {
     return make_double2(fma(a.x, b.x, -__dmul_rn(a.y, b.y)), fma(a.x, b.y, __dmul_rn(a.y, b.x)));
}
// both arrays' value times one complex factor
template <class V> __device__ __forceinline__ PV<V> pcmul(PV<V> a, V w) {
     const V wr = pdup(w.x), wi = pdup(w.y), ni = pdup(-w.y);
     return PV<V>{pfma(a.im, ni, pmul(a.re, wr)), pfma(a.im, wr, pmul(a.re, wi))};
}

// forward 4-point DFT in place, natural-order outputs
template <class V> __device__ __forceinline__ void pdft4(PV<V> &y0, PV<V> &y1, PV<V> &y2, PV<V> &y3) {
     const PV<V> c0 = y0 + y2, c1 = y0 - y2, c2 = y1 + y3, d = y1 - y3;
     y0 = c0 + c2;
     y2 = c0 - c2;
     y1 = PV<V>{padd(c1.re, d.im), psub(c1.im, d.re)};   // c1 - i d
     y3 = PV<V>{psub(c1.re, d.im), padd(c1.im, d.re)};   // c1 + i d
}

// forward 8-point DFT in place, natural-order outputs.  The odd half's
// factors h(1 -+ i), h = sqrt(1/2), are applied in the last additions (fused
// multiply-adds): 52 packed instructions.
template <class V> __device__ __forceinline__ void pdft8(PV<V> (&v)[8]) {
     using R1 = decltype(V::x);
     const V h = pdup(R1(0.70710678118654752440)), mh = pdup(R1(-0.70710678118654752440));
     PV<V> a0 = v[0] + v[4], b0 = v[0] - v[4];
     PV<V> a1 = v[1] + v[5], b1 = v[1] - v[5];
     PV<V> a2 = v[2] + v[6], b2 = v[2] - v[6];
     PV<V> a3 = v[3] + v[7], b3 = v[3] - v[7];
     pdft4(a0, a1, a2, a3);
     // b1 W8 = h (p + i q), b3 W8^3 = h (r - i s)
     const V p = padd(b1.re, b1.im), q = psub(b1.im, b1.re);
     const V r = psub(b3.im, b3.re), s = padd(b3.re, b3.im);
     const V P = padd(p, r), Q = psub(q, s), R = psub(p, r), S = padd(q, s);
     const PV<V> c0{padd(b0.re, b2.im), psub(b0.im, b2.re)};   // b0 - i b2
     const PV<V> c1{psub(b0.re, b2.im), padd(b0.im, b2.re)};   // b0 + i b2
     v[0] = a0;
     v[2] = a1;
     v[4] = a2;
     v[6] = a3;
     v[1] = PV<V>{pfma(P, h, c0.re), pfma(Q, h, c0.im)};
     v[5] = PV<V>{pfma(P, mh, c0.re), pfma(Q, mh, c0.im)};
     v[3] = PV<V>{pfma(S, h, c1.re), pfma(R, mh, c1.im)};
     v[7] = PV<V>{pfma(S, mh, c1.re), pfma(R, h, c1.im)};
}

template <int R, class V>
__device__ __forceinline__ void ppass_dft(PV<V> (&v)[8]) {
     if (R == 8) {
          pdft8(v);
     } else if (R == 4) {
          pdft4(v[0], v[2], v[4], v[6]);
          pdft4(v[1], v[3], v[5], v[7]);
     } else {
#pragma unroll
          for (int q = 0; q < 4; q++) {
               const PV<V> t = v[q];
               v[q] = t + v[q + 4];
               v[q + 4] = t - v[q + 4];
          }
     }
}

// ------------------------------------------------------------------ pass twiddles
//
// The twiddles of the later Stockham passes of an L-point line, in global
// memory (under 6 KB for every length, read through L1 with consecutive lanes
// on consecutive entries): for each pass of span NS = 8, 64, .. and radix R
// the arrays W^jm, W^2jm, W^4jm (as many as log2 R), W = e^{-2 pi i/(NS R)},
// jm < NS, one after the other.

__host__ __device__ constexpr int pass_radix(int L, int NS) { return L / NS >= 8 ? 8 : L / NS; }
__host__ __device__ constexpr int pass_powers(int R) { return R == 8 ? 3 : (R == 4 ? 2 : 1); }
// entries before the arrays of span NS
__host__ __device__ constexpr int ltw_offset(int L, int NS) {
     return NS <= 8 ? 0 : ltw_offset(L, NS / 8) + pass_powers(pass_radix(L, NS / 8)) * (NS / 8);
}

// A pass's twiddles W^jm, W^2jm, W^4jm of the butterflies a thread owns
// (loaded ahead of the exchange that precedes the pass).
template <class V, int L, int NS> struct PassTw {
     static constexpr int R = pass_radix(L, NS), Q = 8 / R, K = pass_powers(R);
     V w[Q][K];
     __device__ __forceinline__ void load(const V *__restrict__ ltw, int t) {
#pragma unroll
          for (int q = 0; q < Q; q++)
#pragma unroll
               for (int k = 0; k < K; k++) w[q][k] = __ldg(&ltw[ltw_offset(L, NS) + k * NS + (t + q * (L / 8)) % NS]);
     }
};

// applied to the T templates whose lines a thread holds
template <int L, int NS, int T, class V>
__device__ __forceinline__ void ppass_twiddle(PV<V> (&v)[T][8], const PassTw<V, L, NS> &tw) {
     constexpr int R = pass_radix(L, NS);
#pragma unroll
     for (int q = 0; q < 8 / R; q++) {
          V w[8];
          w[1] = tw.w[q][0];
          if constexpr (R >= 4) {
               w[2] = tw.w[q][1];
               w[3] = cmul_tw(w[1], w[2]);
          }
          if constexpr (R == 8) {
               w[4] = tw.w[q][2];
               w[5] = cmul_tw(w[1], w[4]);
               w[6] = cmul_tw(w[2], w[4]);
               w[7] = cmul_tw(w[3], w[4]);
          }
#pragma unroll
          for (int r = 1; r < R; r++)
#pragma unroll
               for (int k = 0; k < T; k++) v[k][q + r * (8 / R)] = pcmul(v[k][q + r * (8 / R)], w[r]);
     }
}

// ------------------------------------------------------------------ line transforms
//
// Exchanges through shared memory, position p of a line at p + p/8.
//
// Columns (ROW = false): the lanes of a warp are consecutive t of one line; a
// line holds 16-byte elements (one P2), and a thread holds its T templates'
// lines, BYTES apart.  A 16-byte access is served 8 lanes at a time; the
// padding puts every store and load pattern of the passes on 8 different
// 16-byte banks.
//
// Rows (ROW = true): the lanes are 4 pairs of lines at 8 consecutive t; a
// thread holds the two lines of its pair, the even one first for even t and
// the odd one first for odd t (so that the reads of freshly copied rows,
// 16-byte elements [n2][row], hit 8 different banks).  For the exchanges
// lines hold the real and the imaginary pairs in two planes of 8-byte
// elements, served 16 lanes (4 pairs at 4 t) at a time; lines 2 (mod 16)
// elements apart put those on different banks.

// FP64: 16-byte elements in two planes everywhere, served 8 lanes at a time;
// columns as above, rows 4 lines at 2 consecutive t (lines 2 (mod 8) elements
// apart).

template <class V, int L, bool ROW> struct SplitLine {
     // elements between lines: a value (split-form columns) or one component in each plane
     static constexpr int STRIDE = L + L / 8 + (ROW ? 2 : 0);
     static constexpr int PLANE = (ROW ? run_of<V> : 1) * STRIDE;
     static constexpr bool WHOLE = !ROW && sizeof(V) == 8;   // one 16-byte element per value
     static __device__ __forceinline__ int pos(int p) { return p + (p >> 3); }
     // distance of positions d apart, d a multiple of 8
     static __host__ __device__ constexpr int dist(int d) { return d + d / 8; }
     // bytes of a column line, of the rows of a block
     static constexpr size_t BYTES = 2 * sizeof(V) * (size_t)PLANE;

     static __device__ __forceinline__ void put(unsigned char *s, int p, PV<V> a) {
          if constexpr (WHOLE) {
               reinterpret_cast<float4 *>(s)[p] = pack4(a);
          } else {
               V *f = reinterpret_cast<V *>(s) + p;
               f[0] = a.re;
               f[PLANE] = a.im;
          }
     }
     static __device__ __forceinline__ PV<V> get(const unsigned char *s, int p) {
          if constexpr (WHOLE) {
               return unpack4(reinterpret_cast<const float4 *>(s)[p]);
          } else {
               const V *f = reinterpret_cast<const V *>(s) + p;
               return PV<V>{f[0], f[PLANE]};
          }
     }
};

// the NT threads of a group (one column, one row block) wait for one another
// (id: the group's number within the CTA)
template <int NT>
__device__ __forceinline__ void group_sync(int id) {
     if (NT <= 32)
          __syncwarp();
     else
          asm volatile("bar.sync %0, %1;" ::"r"(id + 1), "n"(NT > 32 ? NT : 32) : "memory");
}
// threads of a group: L/8 per column, four times that per row block
template <int L, bool ROW> constexpr int group_threads = ROW ? L / 2 : L / 8;

// The passes from span NS on, the data and the pass's twiddles at hand, by a
// group of NT threads.  s: the memory of the thread's first line, the k-th
// one's `next` bytes further; read() is called when the thread has read the
// last exchange; threads with active = false only keep the group's barriers.
template <int L, bool ROW, int NS, int NT, int T, class V, class F>
__device__ __forceinline__ void line_pass(PV<V> (&v)[T][8], unsigned char *s, int next, const V *__restrict__ ltw,
                                          int t, int id, const PassTw<V, L, (NS > 1 ? NS : 8)> &tw, const F &read,
                                          bool active) {
     using G = SplitLine<V, L, ROW>;
     constexpr int R = pass_radix(L, NS);
     if (active) {
          if constexpr (NS > 1) ppass_twiddle<L, NS, T>(v, tw);
#pragma unroll
          for (int k = 0; k < T; k++) ppass_dft<R>(v[k]);
     }
     if constexpr (NS * R < L) {
          // (R = 8 here) output r of butterfly t goes to (t/NS)*8 NS + t%NS + r NS
          constexpr int RN = pass_radix(L, NS * 8);
          PassTw<V, L, NS * 8> tn;
          if (active) tn.load(ltw, t);
          if constexpr (NS > 1) group_sync<NT>(id);   // the previous exchange is read
          const int d = NS == 1 ? G::dist(8) * t : G::pos((t / NS) * NS * 8 + (t % NS));
          if (active) {
#pragma unroll
               for (int k = 0; k < T; k++)
#pragma unroll
                    for (int r = 0; r < 8; r++) G::put(s + k * next, d + (NS == 1 ? r : r * G::dist(NS)), v[k][r]);
          }
          group_sync<NT>(id);
          if (active) {
#pragma unroll
               for (int k = 0; k < T; k++)
#pragma unroll
                    for (int q = 0; q < 8 / RN; q++) {
                         const int d1 = G::pos(t + q * (L / 8));
#pragma unroll
                         for (int r = 0; r < RN; r++)
                              v[k][q + r * (8 / RN)] = G::get(s + k * next, d1 + r * G::dist(L / RN));
                    }
          }
          if constexpr (NS * 8 * RN >= L) read();
          line_pass<L, ROW, NS * 8, NT, T>(v, s, next, ltw, t, id, tn, read, active);
     }
}

// L-point forward transform of a thread's T lines: thread t holds
// x[t + m L/8] on entry and X[t + m L/8] on exit.  The lines' shared memory
// must be free on entry.
template <int L, bool ROW, int T, int NT = group_threads<L, ROW>, class V, class F>
__device__ __forceinline__ void split_fft(PV<V> (&v)[T][8], unsigned char *s, int next, const V *__restrict__ ltw,
                                          int t, int id, const F &read, bool active = true) {
     line_pass<L, ROW, 1, NT, T>(v, s, next, ltw, t, id, PassTw<V, L, 8>(), read, active);
}

// ------------------------------------------------------------------ column pass

struct SplitCol {
     const float4 *xab;      // operands, layout above
     const float *s2;
     const TmplParam *tp;
     float4 *y;
     const float2 *w0;       // W^(n2 t) [N2][L/8], W = e^{-2 pi i/nfftf}
     const float2 *ws;       // W^(n2 L/8) [N2]
     const float2 *ltw;      // pass twiddles of an L-point line
     int N;                  // samples
     int CL;                 // entries per operand column (a multiple of 32, zero past the last sample)
     int rows;               // ceil(N / N2)
     int nifo;
     int nt;                 // templates of the launch
};

// x (c - i s) for both arrays
__device__ __forceinline__ P2 rot1(const float4 x, float ph) {
     float sn, cs;
     __sincosf(ph, &sn, &cs);
     const P2 a = unpack4(x);
     const float2 c = pdup(cs), s = pdup(sn), ns = pdup(-sn);
     return P2{pfma(a.re, c, pmul(a.im, s)), pfma(a.im, c, pmul(a.re, ns))};
}

// x0 (c0 - i s0) + x1 (c1 - i s1), one chain of fused multiply-adds per component
__device__ __forceinline__ P2 rot2(const float4 x0, const float4 x1, float ph0, float ph1) {
     float s0, c0, s1, c1;
     __sincosf(ph0, &s0, &c0);
     __sincosf(ph1, &s1, &c1);
     const P2 a = unpack4(x0), b = unpack4(x1);
     const float2 C0 = pdup(c0), S0 = pdup(s0), M0 = pdup(-s0), C1 = pdup(c1), S1 = pdup(s1), M1 = pdup(-s1);
     return P2{pfma(a.re, C0, pfma(a.im, S0, pfma(b.re, C1, pmul(b.im, S1)))),
               pfma(a.im, C0, pfma(a.re, M0, pfma(b.im, C1, pmul(b.re, M1))))};
}

// Compensated accumulation of both arrays' network sum: c collects the exact
// rounding error of every addition (two-sum), as Neumaier's sum does.
struct PCompSum {
     float2 s, c;
     __device__ __forceinline__ void init(float2 v) { s = v; c = pdup(0.f); }
     __device__ __forceinline__ void add(float2 x) {
          const float2 t = padd(s, x), z = psub(t, s);
          c = padd(c, padd(psub(s, psub(t, z)), psub(x, z)));
          s = t;
     }
     __device__ __forceinline__ float2 value() const { return padd(s, c); }
};

// The operands of one sample: every detector's x and 2 i shft.
template <int NIFO> struct SampleOps {
     float4 x[NIFO];
     float s[NIFO];
};

// loads kept where they are written (volatile): issued ahead of their use
__device__ __forceinline__ float4 ldg4_v(const float4 *p) {
     float4 q;
     asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(q.x), "=f"(q.y), "=f"(q.z), "=f"(q.w) : "l"(p));
     return q;
}
__device__ __forceinline__ float2 ldg2_v(const float *p) {
     float2 q;
     asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];" : "=f"(q.x), "=f"(q.y) : "l"(p));
     return q;
}
__device__ __forceinline__ float ldg1_v(const float *p) {
     float q;
     asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(q) : "l"(p));
     return q;
}

template <int NIFO>
__device__ __forceinline__ void load_ops(SampleOps<NIFO> &o, const float4 *x, const float *s, size_t plane) {
#pragma unroll
     for (int d = 0; d < NIFO; d++) o.x[d] = ldg4_v(x + d * plane);
     if constexpr (NIFO == 2) {
          const float2 q = ldg2_v(s);
          o.s[0] = q.x;
          o.s[1] = q.y;
     } else {
#pragma unroll
          for (int d = 0; d < NIFO; d++) o.s[d] = ldg1_v(s + d);
     }
}

// The spindown phase het1*i + spnd*i^2 of a template, formed and reduced in
// FP64.  In turns it is q*i with q = h + w*i; one fused multiply-add onto
// 1.5*2^20 leaves the fraction of a turn, to 2^-33, in the low word as a
// signed 32-bit number (the FP64 <-> integer conversions and rint that this
// replaces ran at a quarter of the multiply-adds' rate).  Phases of 2^18
// turns and more (BIG) have their whole turns taken off first.
//
// The number has more digits than a float: its upper 24 bits and its lower 8
// are taken separately (both exact), and 2 pi/2^32 in two floats, so that the
// radians are rounded to FP32 once, by the last multiply-add.  Errors over 6000
// samples of six days: at most 1.2e-7 rad, rms 4.5e-8, as from FP64 radians
// (with the whole number converted and multiplied at once 2.8e-7, 7.6e-8).
// Column pass with this and without: 1.40 and 1.42 us per template of 2^18
// points, 0.777 and 0.776 of 2^17; one detector 0.737 and 0.726, three (2^18)
// 1.655 and 1.624.
struct SpinPhase {
     double h, w;   // het1, spnd in turns
     // returns whether some sample's phase may reach 2^18 turns
     __host__ __device__ __forceinline__ bool init(double het1, double spnd, int N) {
          h = het1 * INV_TWO_PI;
          w = spnd * INV_TWO_PI;
          return !((fabs(h) + fabs(w) * (double)N) * (double)N < 262144.);
     }
     // radians in [-pi, pi]; di = (double)i
     template <bool BIG>
     __host__ __device__ __forceinline__ float at(double di) const {
          const double q = fma(w, di, h);
          double c = 1572864.;
          if (BIG) {
               const double r = 6755399441055744.;   // 1.5*2^52
               c = dsub(c, dsub(dadd(q * di, r), r));
          }
          const int n = low_word(fma(q, di, c));
          constexpr double rad = TWO_PI / 4294967296.;
          constexpr float r1 = (float)rad, r2 = (float)(rad - (double)r1);
          const float up = (float)(n & ~255);
          const float lo = fmaf(float_of_bits((unsigned)(n & 255) | 0x4b000000u), r1, -8388608.f * r1);   // (2^23 + low bits - 2^23) r1
          return fmaf(up, r1, fmaf(up, r2, lo));
     }
};

// The spindown modulation (spinmod.c:490-514) of one sample: the phase pr,
// plus spnd*(2 i shft_n[i]) in FP32 per detector; FP32 sincos and products.
// The network sum is compensated for three or more detectors; for one or two
// it is a single rounded addition, which compensation would not change.
template <int NIFO>
__device__ __forceinline__ P2 demod_sample(const SampleOps<NIFO> &o, float pr, float spf) {
     if constexpr (NIFO == 1) {
          return rot1(o.x[0], fmaf(spf, o.s[0], pr));
     } else if constexpr (NIFO == 2) {
          return rot2(o.x[0], o.x[1], fmaf(spf, o.s[0], pr), fmaf(spf, o.s[1], pr));
     } else {
          PCompSum re, im;
#pragma unroll
          for (int d = 0; d < NIFO; d++) {
               const P2 p = rot1(o.x[d], fmaf(spf, o.s[d], pr));
               if (d == 0) {
                    re.init(p.re);
                    im.init(p.im);
               } else {
                    re.add(p.re);
                    im.add(p.im);
               }
          }
          return P2{re.value(), im.value()};
     }
}

// the same with the detector count read at run time (more than three)
__device__ __forceinline__ P2 demod_sample_n(const float4 *x, const float *s, size_t plane, int nifo, float pr, float spf) {
     PCompSum re, im;
     for (int d = 0; d < nifo; d++) {
          const P2 p = rot1(__ldg(x + d * plane), fmaf(spf, __ldg(s + d), pr));
          if (d == 0) {
               re.init(p.re);
               im.init(p.im);
          } else {
               re.add(p.re);
               im.add(p.im);
          }
     }
     return P2{re.value(), im.value()};
}

// What split_demod() works from: the T templates' phases and operands.
template <int T> struct DemodIn {
     const float4 *xp[T];
     const float *sp[T];
     SpinPhase ph[T];
     float spf[T];
     double d0;       // sample number of m = 0
     size_t plane;    // operands of one detector and slot
};

// The first MC samples m of a thread, its templates sharing their operands;
// straight-line code, so that several samples' chains (FP64 phase, sine and
// cosine, rotation) are in flight.  The loads of sample m + AHEAD are issued
// before sample m is worked on.
template <int L, int N2, int NIFO, int T, int MC>
__device__ __forceinline__ void demod_run(P2 (&v)[T][8], const DemodIn<T> &in) {
     constexpr int AHEAD = 2;
     SampleOps<NIFO> o[MC];
#pragma unroll
     for (int m = 0; m < AHEAD && m < MC; m++)
          load_ops<NIFO>(o[m], in.xp[0] + m * (L / 8), in.sp[0] + m * (L / 8) * NIFO, in.plane);
#pragma unroll
     for (int m = 0; m < MC; m++) {
          if (m + AHEAD < MC)
               load_ops<NIFO>(o[(m + AHEAD) % MC], in.xp[0] + (m + AHEAD) * (L / 8),
                              in.sp[0] + (m + AHEAD) * (L / 8) * NIFO, in.plane);
          const double di = in.d0 + (double)(m * (N2 * (L / 8)));
#pragma unroll
          for (int k = 0; k < T; k++) v[k][m] = demod_sample<NIFO>(o[m], in.ph[k].template at<false>(di), in.spf[k]);
     }
#pragma unroll
     for (int m = MC; m < 8; m++)
#pragma unroll
          for (int k = 0; k < T; k++) v[k][m] = pzero();
}

// The eight samples n1 = t + m L/8 of column n2 for the T templates b0 ..
// b0+T-1.  Templates of one sky point (the spindowns that follow one another)
// share the operands.  Operand columns are zero past the last sample, and
// warps wholly past it (i.e. past row a.rows) skip.
template <int L, int N2, int NIFO, int T>
__device__ __forceinline__ void split_demod(P2 (&v)[T][8], const SplitCol &a, int b0, int n2, int t) {
     const int nf = NIFO > 0 ? NIFO : a.nifo;
     DemodIn<T> in;
     in.plane = (size_t)N2 * a.CL;
     in.d0 = (double)(N2 * t + n2);
     bool plain = true;
#pragma unroll
     for (int k = 0; k < T; k++) {
          const TmplParam P = a.tp[min(b0 + k, a.nt - 1)];
          if (in.ph[k].init(P.het1, P.spnd, a.N)) plain = false;
          in.spf[k] = (float)P.spnd;
          in.xp[k] = a.xab + ((size_t)P.slot * nf * N2 + n2) * a.CL + t;
          in.sp[k] = a.s2 + (((size_t)P.slot * N2 + n2) * a.CL + t) * nf;
          if (in.xp[k] != in.xp[0]) plain = false;
     }
     const int wt = L / 8 >= 32 ? (t & ~31) : 0;   // the warp's first t
     const int mc = (a.rows - wt + L / 8 - 1) / (L / 8);   // samples m < mc lie before the last row
     if constexpr (NIFO > 0) {
          if (plain) {
               if (mc >= 8) return demod_run<L, N2, NIFO, T, 8>(v, in);
               if (mc == 7) return demod_run<L, N2, NIFO, T, 7>(v, in);
               if (mc == 6) return demod_run<L, N2, NIFO, T, 6>(v, in);
               if (mc == 5) return demod_run<L, N2, NIFO, T, 5>(v, in);
               if (mc == 4) return demod_run<L, N2, NIFO, T, 4>(v, in);
          }
     }
     // templates of different sky points, phases past 2^18 turns, few rows,
     // more than three detectors
#pragma unroll
     for (int m = 0; m < 8; m++) {
          const double di = in.d0 + (double)(m * (N2 * (L / 8)));
#pragma unroll
          for (int k = 0; k < T; k++) {
               v[k][m] = pzero();
               if (m < mc) {
                    const float4 *x = in.xp[k] + m * (L / 8);
                    const float *s = in.sp[k] + m * (L / 8) * nf;
                    const float pr = in.ph[k].template at<true>(di);
                    if constexpr (NIFO > 0) {
                         SampleOps<NIFO> o;
                         load_ops<NIFO>(o, x, s, in.plane);
                         v[k][m] = demod_sample<NIFO>(o, pr, in.spf[k]);
                    } else {
                         v[k][m] = demod_sample_n(x, s, in.plane, nf, pr, in.spf[k]);
                    }
               }
          }
     }
}

// column n2 of templates b0 .. b0+T-1 (below a.nt) by the threads t < L/8 of
// one group; s: the group's line memory
template <int L, int N2, int NIFO, int T>
__device__ __forceinline__ void split_col_line(const SplitCol &a, int b0, int n2, int t, int line, unsigned char *s) {
     P2 v[T][8];
     split_demod<L, N2, NIFO, T>(v, a, b0, n2, t);
     float2 w = __ldg(&a.w0[n2 * (L / 8) + t]);
     const float2 st = __ldg(&a.ws[n2]);
     split_fft<L, false, T>(v, s, (int)SplitLine<float2, L, false>::BYTES, a.ltw, t, line, [] {});
     // times W^(n2 k1), k1 = t + m L/8, by recurrence from the base twiddle
     // (seven products: relative error below 1e-6)
     float4 *dst = a.y + (size_t)b0 * (L * N2) + ((size_t)(t / RUN) * N2 + n2) * RUN + t % RUN;
#pragma unroll
     for (int m = 0; m < 8; m++) {
          if (m > 0) w = cmul_tw(w, st);
#pragma unroll
          for (int k = 0; k < T; k++)
               if (k == 0 || b0 + k < a.nt)
                    dst[(size_t)k * (L * N2) + (size_t)m * (L / 8) * N2] = pack4(pcmul(v[k][m], w));
     }
}

// columns per CTA: CTAs of at most 256 threads (the shortest columns: 64),
// so that the last wave of a launch and small launches are spread well
template <int L> __host__ __device__ constexpr int split_col_lines() { return L >= 1024 ? 2 : (L >= 512 ? 4 : 8); }

template <int L> __host__ __device__ constexpr int split_col_threads() { return split_col_lines<L>() * L / 8; }
// resident CTAs per SM: 32 warps of 64 registers (T = 1), 16 of 128 (T = 2)
template <int L, int T> __host__ __device__ constexpr int split_col_blocks() { return 1024 / T / split_col_threads<L>(); }

// grid (N2 / split_col_lines<L>(), ceil(templates / T))
template <int L, int N2, int NIFO, int T>
__global__ void __launch_bounds__(split_col_threads<L>(), split_col_blocks<L, T>())
k_split_col(const __grid_constant__ SplitCol a) {
     extern __shared__ __align__(128) unsigned char smem_raw[];
     const int line = threadIdx.x / (L / 8), t = threadIdx.x % (L / 8);
     split_col_line<L, N2, NIFO, T>(a, blockIdx.y * T, blockIdx.x * split_col_lines<L>() + line, t, line,
                                    smem_raw + line * (T * SplitLine<float2, L, false>::BYTES));
}

// ------------------------------------------------------------------ column pass, FP64 form

struct Fp64Col {
     const double2 *xre, *xim;   // operands (a.re, b.re), (a.im, b.im), layout above
     const double *t1;           // i^2 + 2 i shft_n[i]
     const TmplParam *tp;
     double2 *y;
     const double2 *w0;          // W^(n2 t) [N2][L/8], W = e^{-2 pi i/nfftf}
     const double2 *ws;          // W^(n2 m L/8) [N2][8]
     const double2 *ltw;         // pass twiddles of an L-point line
     int CL;                     // entries per operand column (a multiple of 32, zero past the last sample)
     int rows;                   // ceil(N / N2)
     int N2, nifo;
};

// sin and cos of the spindown phase, |x| < 2^30 rad: reduced by multiples of
// pi/2 (two fused multiply-adds), then the Taylor series on [-pi/4, pi/4] up to
// x^17 and x^16 (remainders below 3e-18).  The error is absolute, as a factor of
// the demodulation needs it: below 2^-52 (1.3e-16 measured, rms 3.17e-17;
// sincos() 1.3e-16 and 3.18e-17 over the same 2^20 phases up to 1e9 rad).
// Relative to a value near zero it may be large.  Without the library's
// argument checks and branches, so that several samples' chains are in flight.
__host__ __device__ __forceinline__ void sincos_spin(double x, double &sn, double &cs) {
     const double big = 6755399441055744.;   // 1.5*2^52
     const double kb = fma(x, 0.63661977236758134308, big);
     const int q = low_word(kb);
     const double k = dsub(kb, big);
     double r = fma(-k, 1.5707963267948965580, x);
     r = fma(-k, 6.1232339957367660359e-17, r);
     const double z = r * r;
     double p = fma(z, 1. / 355687428096000., -1. / 1307674368000.);
     p = fma(z, p, 1. / 6227020800.);
     p = fma(z, p, -1. / 39916800.);
     p = fma(z, p, 1. / 362880.);
     p = fma(z, p, -1. / 5040.);
     p = fma(z, p, 1. / 120.);
     p = fma(z, p, -1. / 6.);
     const double s = fma(r * z, p, r);
     p = fma(z, 1. / 20922789888000., -1. / 87178291200.);
     p = fma(z, p, 1. / 479001600.);
     p = fma(z, p, -1. / 3628800.);
     p = fma(z, p, 1. / 40320.);
     p = fma(z, p, -1. / 720.);
     p = fma(z, p, 1. / 24.);
     p = fma(z, p, -1. / 2.);
     const double c = fma(z, p, 1.);
     const double a = q & 1 ? c : s, b = q & 1 ? s : c;
     sn = q & 2 ? -a : a;
     cs = (q + 1) & 2 ? -b : b;
}
__device__ __noinline__ void sincos_large(double x, double *s, double *c) { sincos(x, s, c); }

__device__ __forceinline__ double2 ldgd2_v(const double2 *p) {
     double2 q;
     asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(q.x), "=d"(q.y) : "l"(p));
     return q;
}
__device__ __forceinline__ double ldgd_v(const double *p) {
     double q;
     asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(q) : "l"(p));
     return q;
}

// acc + (re + i im) (c - i s) for both arrays
__device__ __forceinline__ D2 rot64(const double2 re, const double2 im, double sn, double cs, D2 acc) {
     const double2 C = pdup(cs), S = pdup(sn), M = pdup(-sn);
     return D2{pfma(re, C, pfma(im, S, acc.re)), pfma(im, C, pfma(re, M, acc.im))};
}

// Samples n1 = t + m L/8, m < 8, of column n2 for template P: the reference's
// DOUBLE-build spindown_modulation (spinmod.c:490-514), the phase het1*i +
// spnd*t1 with its products and sum rounded as there.  fp64_run() takes the
// first MC in straight-line code, the operands of the next sample loaded
// before one is worked on (without: 4.3 of 9 cycles per instruction waiting
// for loads, 5.0 us per template of 2^18 points); it returns whether a phase
// reached 2^30 rad.
struct Fp64In {
     const double2 *xre, *xim;
     const double *t1;
     size_t plane;     // operands of one detector
     double d0, dm;    // sample number of m = 0, step in m
};

template <int L, int NIFO, int MC>
__device__ __forceinline__ bool fp64_run(D2 (&v)[8], const Fp64In &in, const TmplParam &P) {
     double2 re[2][NIFO], im[2][NIFO];
     double t1[2][NIFO];
     double far = 0.;
     auto load = [&](int m) {
#pragma unroll
          for (int d = 0; d < NIFO; d++) {
               const size_t e = d * in.plane + m * (L / 8);
               re[m & 1][d] = ldgd2_v(&in.xre[e]);
               im[m & 1][d] = ldgd2_v(&in.xim[e]);
               t1[m & 1][d] = ldgd_v(&in.t1[e]);
          }
     };
     load(0);
#pragma unroll
     for (int m = 0; m < MC; m++) {
          if (m + 1 < MC) load(m + 1);
          const double hi = __dmul_rn(P.het1, in.d0 + m * in.dm);
          v[m] = pzero_of<double2>();
#pragma unroll
          for (int d = 0; d < NIFO; d++) {
               const double x = __dadd_rn(hi, __dmul_rn(P.spnd, t1[m & 1][d]));
               far = fmax(far, fabs(x));
               double sn, cs;
               sincos_spin(x, sn, cs);
               v[m] = rot64(re[m & 1][d], im[m & 1][d], sn, cs, v[m]);
          }
     }
#pragma unroll
     for (int m = MC; m < 8; m++) v[m] = pzero_of<double2>();
     return !(far < 1073741824.);
}

template <int L, int NIFO>
__device__ __forceinline__ void fp64_demod(D2 (&v)[8], const Fp64Col &a, const TmplParam &P, int n2, int t) {
     const int nf = NIFO > 0 ? NIFO : a.nifo;
     Fp64In in;
     in.plane = (size_t)a.N2 * a.CL;
     const size_t o = ((size_t)P.slot * nf * a.N2 + n2) * a.CL + t;
     in.xre = a.xre + o;
     in.xim = a.xim + o;
     in.t1 = a.t1 + o;
     in.d0 = (double)(a.N2 * t + n2);
     in.dm = (double)(a.N2 * (L / 8));
     const int wt = L / 8 >= 32 ? (t & ~31) : 0;   // the warp's first t
     const int mc = (a.rows - wt + L / 8 - 1) / (L / 8);   // samples m < mc lie before the last row
     bool far = true;
     if constexpr (NIFO > 0) {
          if (mc >= 8) far = fp64_run<L, NIFO, 8>(v, in, P);
          else if (mc == 7) far = fp64_run<L, NIFO, 7>(v, in, P);
          else if (mc == 6) far = fp64_run<L, NIFO, 6>(v, in, P);
          else if (mc == 5) far = fp64_run<L, NIFO, 5>(v, in, P);
          else if (mc == 4) far = fp64_run<L, NIFO, 4>(v, in, P);
     }
     if (!far) return;
     // phases past 2^30 rad, few rows, more than three detectors
#pragma unroll
     for (int m = 0; m < 8; m++) {
          v[m] = pzero_of<double2>();
          if (m < mc) {
               const double hi = __dmul_rn(P.het1, in.d0 + m * in.dm);
               for (int d = 0; d < nf; d++) {
                    const size_t e = d * in.plane + m * (L / 8);
                    const double x = __dadd_rn(hi, __dmul_rn(P.spnd, __ldg(&in.t1[e])));
                    double sn, cs;
                    if (fabs(x) < 1073741824.) sincos_spin(x, sn, cs);
                    else sincos_large(x, &sn, &cs);
                    v[m] = rot64(__ldg(&in.xre[e]), __ldg(&in.xim[e]), sn, cs, v[m]);
               }
          }
     }
}

// columns per CTA (256 threads, the shortest columns 64)
template <int L> __host__ __device__ constexpr int fp64_col_lines() { return L >= 512 ? 4 : 8; }
template <int L> __host__ __device__ constexpr int fp64_col_threads() { return fp64_col_lines<L>() * L / 8; }

// grid (N2 / fp64_col_lines<L>(), templates); 16 warps of 128 registers per SM
template <int L, int NIFO>
__global__ void __launch_bounds__(fp64_col_threads<L>(), 512 / fp64_col_threads<L>())
k_fp64_col(const __grid_constant__ Fp64Col a) {
     extern __shared__ __align__(128) unsigned char smem_raw[];
     using G = SplitLine<double2, L, false>;
     constexpr int R = run_of<double2>;
     const int line = threadIdx.x / (L / 8), t = threadIdx.x % (L / 8);
     const int n2 = blockIdx.x * fp64_col_lines<L>() + line, b = blockIdx.y;
     const TmplParam P = a.tp[b];
     D2 v[1][8];
     fp64_demod<L, NIFO>(v[0], a, P, n2, t);
     split_fft<L, false, 1>(v, smem_raw + line * G::BYTES, 0, a.ltw, t, line, [] {});
     // times W^(n2 k1), k1 = t + m L/8: one product of table entries each
     const double2 w = __ldg(&a.w0[n2 * (L / 8) + t]);
     double2 *dst = a.y + ((size_t)b * (L / R) + t / R) * (2 * R * a.N2) + n2 * R + t % R;
#pragma unroll
     for (int m = 0; m < 8; m++) {
          const D2 q = pcmul(v[0][m], m == 0 ? w : cmul_tw(w, __ldg(&a.ws[n2 * 8 + m])));
          double2 *d = dst + (size_t)m * (L / 8 / R) * (2 * R * a.N2);
          d[0] = q.re;
          d[R * a.N2] = q.im;
     }
}

// ------------------------------------------------------------------ row pass

// Candidate records of the sparse F store (16 bytes): template (within the
// resolve group) | kind << 24, bin, F[bin], and one neighbour's F.
constexpr unsigned CAND_LOCAL = 0u;   // a local maximum decided in the row pass; no tie with bin-1
constexpr unsigned CAND_LEFT = 1u;    // first bin of a CTA's run: F[bin-1] is in the edge ring (nb = F[bin+1])
constexpr unsigned CAND_RIGHT = 2u;   // last bin of a run: F[bin+1] is in the edge ring (nb = F[bin-1])
constexpr unsigned CAND_TIE = 3u;     // F[bin-1] == F[bin]: the MAX_ALG 3 run needs F[bin-2]
constexpr unsigned ERR_NEED_FULL_F = 4u;   // a batch needs the full F spectra (tie or candidate overflow)

// Two ways to hand F to the trigger selection:
//   full (E == nullptr): the whole spectrum [fr0, fr1] goes to the F ring
//     and the bins passing the threshold test to the candidate list (uint2
//     {template, bin}); used with blocks_avg and as the fallback.
//   sparse (E != nullptr): no spectrum leaves the SM.  The RUN lanes c of a
//     thread group hold the consecutive bins k1b + c + N1*k2 of one k2, so a
//     bin's neighbours are one shuffle away except at the run's ends: the
//     row pass decides the local-maximum test itself for the bins between and
//     writes candidate records (uint4, kinds above) for bins passing the
//     threshold; only the end bins c = 0 and RUN-1 of every run go to the
//     edge ring E[((b*NJ + j)*L + k2)*2 + (c > 0)] (j = CTA index) for the
//     neighbours of the other CTAs' end-bin candidates.
template <class W> struct RowArgs {
     using V = W;
     using R1 = decltype(V::x);
     const V *y;
     const V *ltw;
     R1 *F;
     const TmplParam *tp;
     const AaBb *ab;
     int nF, fr0, fr1;
     double thr;
     uint2 *cand;
     unsigned *cand_cnt;
     unsigned cand_cap;
     int boff;        // index of this chunk's first template within its resolve group
     float *E;        // sparse form: edge ring of the resolve group
     uint4 *scand;    // sparse form: candidate records
     int nt;          // templates of the launch
     unsigned *err;
     int probes;      // limit of the waits for a row block
};
using SplitRow = RowArgs<float2>;
using Fp64Row = RowArgs<double2>;

// F = |Fa|^2 * (1/aa) + |Fb|^2 * (1/bb) of the outputs k2 = t + m L/8 of the
// rows k1, k1 + 1 (k1 = RUN blk + 2c, lanes c of a group of 4 adjacent; v[0]
// is row k1 for even t, k1 + 1 for odd t); HALF: only k2 < L/2 (every bin the
// search keeps lies below nfftf/2; the others are dead and never computed).
template <int L, int N1, bool HALF>
__device__ __forceinline__ void split_fstat(const P2 (&v)[2][8], const SplitRow &a, int b, int k1, int t) {
     constexpr int M = HALF ? 4 : 8;
     const AaBb sums = a.ab[a.tp[b].slot];
     const float ia = 1.f / sums.aaf, ib = 1.f / sums.bbf;
     const float thrf = (float)a.thr;
     const bool exact_thr = (double)thrf == a.thr;   // then f < thr compares the same in float
     float f[M][2];
     bool pass[M][2], any = false;
#pragma unroll
     for (int m = 0; m < M; m++) {
          const float2 q = pfma(v[0][m].re, v[0][m].re, pmul(v[0][m].im, v[0][m].im));
          const float2 r = pfma(v[1][m].re, v[1][m].re, pmul(v[1][m].im, v[1][m].im));
          const float f0 = fmaf(q.x, ia, q.y * ib), f1 = fmaf(r.x, ia, r.y * ib);
          f[m][0] = t & 1 ? f1 : f0;
          f[m][1] = t & 1 ? f0 : f1;
#pragma unroll
          for (int j = 0; j < 2; j++) {
               const int k = k1 + j + N1 * (t + m * (L / 8));
               pass[m][j] = (exact_thr ? !(f[m][j] < thrf) : !((double)f[m][j] < a.thr)) && k >= a.fr0 + 1 && k < a.fr1 - 1;
               any |= pass[m][j];
          }
     }
     const unsigned bg = (unsigned)(b + a.boff);
     if (a.E == nullptr) {
          float *dst = a.F + (size_t)b * a.nF - a.fr0;
#pragma unroll
          for (int m = 0; m < M; m++)
#pragma unroll
               for (int j = 0; j < 2; j++) {
                    const int k = k1 + j + N1 * (t + m * (L / 8));
                    if (k >= a.fr0 && k <= a.fr1) dst[k] = f[m][j];
                    if (a.cand && pass[m][j]) {
                         const unsigned c = atomicAdd(a.cand_cnt, 1u);
                         if (c < a.cand_cap) a.cand[c] = make_uint2(bg, (unsigned)k);
                    }
               }
          return;
     }
     const int c = k1 % RUN;   // 0, 2, .. RUN - 2
     if (c == 0 || c == RUN - 2) {
          const int e = c == 0 ? 0 : 1;   // the run's first or last bin
          float *ej = a.E + ((size_t)bg * (N1 / RUN) + k1 / RUN) * (2 * L) + e;
#pragma unroll
          for (int m = 0; m < M; m++) {
               const int k2 = t + m * (L / 8), k = k1 + e + N1 * k2;
               if (k >= a.fr0 && k <= a.fr1) ej[2 * k2] = e == 0 ? f[m][0] : f[m][1];
          }
     }
     // bins over the threshold are rare: look at neighbours only in warps that hold one
     if (!__any_sync(0xffffffffu, any)) return;
#pragma unroll
     for (int m = 0; m < M; m++) {
          // the neighbouring bins of the pair within the run (the next lanes of the same k2)
          const float below = __shfl_up_sync(0xffffffffu, f[m][1], 1, RUN / 2);
          const float above = __shfl_down_sync(0xffffffffu, f[m][0], 1, RUN / 2);
#pragma unroll
          for (int j = 0; j < 2; j++) {
               if (!pass[m][j]) continue;
               const float g = f[m][j], fm = j == 0 ? below : f[m][0], fp = j == 0 ? f[m][1] : above;
               const int k = k1 + j + N1 * (t + m * (L / 8));
               unsigned kind;
               float nb = 0.f;
               bool keep = true;
               if (c + j == 0) {
                    kind = CAND_LEFT;
                    nb = fp;
               } else if (c + j == RUN - 1) {
                    kind = CAND_RIGHT;
                    nb = fm;
               } else {
                    keep = !(fm > g || g < fp);   // a local maximum
                    kind = fm == g ? CAND_TIE : CAND_LOCAL;
               }
               if (keep) {
                    const unsigned q = atomicAdd(a.cand_cnt, 1u);
                    if (q < a.cand_cap)
                         a.scand[q] = make_uint4(bg | (kind << 24), (unsigned)k, __float_as_uint(g), __float_as_uint(nb));
               }
          }
     }
}

// rows k1 = RUN blk .. RUN blk + 7 of template b, thread (c, t) = (tid % 4,
// tid / 4) of the group on rows 2c and 2c + 1; y: element (n2 = 0, row 0)
// of the CTA's rows, in shared (copied by the caller) or global memory
template <int L, int N1, bool HALF, class F>
__device__ __forceinline__ void split_row_block(const SplitRow &a, int b, int blk, int tid, int id, const float2 *y,
                                                bool shared, unsigned char *lines, const F &read) {
     constexpr int LB = 8 * SplitLine<float2, L, true>::STRIDE;   // bytes between lines in a plane
     const int c = tid % (RUN / 2), t = tid / (RUN / 2), odd = t & 1;
     const float4 *src = reinterpret_cast<const float4 *>(y) + t * RUN + 2 * c + odd;
     P2 v[2][8];
#pragma unroll
     for (int m = 0; m < 8; m++) {
          const float4 *p = src + m * (L / 8 * RUN);
          v[0][m] = unpack4(shared ? p[0] : __ldcg(p));
          v[1][m] = unpack4(shared ? p[1 - 2 * odd] : __ldcg(p + 1 - 2 * odd));
     }
     if (shared) group_sync<L / 2>(id);   // the exchanges reuse the rows' memory
     split_fft<L, true, 2>(v, lines + (2 * c + odd) * LB, LB * (1 - 2 * odd), a.ltw, t, id, read);
     split_fstat<L, N1, HALF>(v, a, b, blk * RUN + 2 * c, t);
}

// F = A/aa + B/bb of the FP64 form (A = |Fa|^2, B = |Fb|^2) with 1/aa and 1/bb
// in two doubles each, whose lower parts' terms are added first: two roundings
// of F's size, where the two quotients and their sum make three.  Row pass at
// 2^18 points 2.35 us per template, with divisions 2.51 (2.28 with single
// reciprocals, which round once more than the divisions).
struct FstatSums {
     double aa, bb, ah, al, bh, bl;
     __host__ __device__ __forceinline__ FstatSums(double a, double b) : aa(a), bb(b), ah(1. / a), bh(1. / b) {
          al = fma(-ah, aa, 1.) * ah;
          bl = fma(-bh, bb, 1.) * bh;
     }
     __host__ __device__ __forceinline__ double f(double A, double B) const {
          const double v = fma(A, ah, fma(B, bh, fma(A, al, B * bl)));
          // sums that are zero, values that are not finite
          return fabs(v) <= DBL_MAX ? v : A / aa + B / bb;
     }
};

// F of row k1 in the FP64 form, the full store (see RowArgs), HALF as above
template <int L, int N1, bool HALF>
__device__ __forceinline__ void fp64_fstat(const D2 (&v)[8], const Fp64Row &a, int b, int k1, int t) {
     const AaBb ab = a.ab[a.tp[b].slot];
     const FstatSums sums(ab.aa, ab.bb);
     double *dst = a.F + (size_t)b * a.nF - a.fr0;
#pragma unroll
     for (int m = 0; m < (HALF ? 4 : 8); m++) {
          const int k = k1 + N1 * (t + m * (L / 8));
          if (k >= a.fr0 && k <= a.fr1) {
               const double2 q = pfma(v[m].re, v[m].re, pmul(v[m].im, v[m].im));
               const double f = sums.f(q.x, q.y);
               dst[k] = f;
               if (a.cand && !(f < a.thr) && k >= a.fr0 + 1 && k < a.fr1 - 1) {
                    const unsigned c = atomicAdd(a.cand_cnt, 1u);
                    if (c < a.cand_cap) a.cand[c] = make_uint2((unsigned)(b + a.boff), (unsigned)k);
               }
          }
     }
}

// the FP64 form's block: rows k1 = 4 blk + c, one line per thread (c, t) = (tid % 4, tid / 4)
template <int L, int N1, bool HALF, class F>
__device__ __forceinline__ void split_row_block(const Fp64Row &a, int b, int blk, int tid, int id, const double2 *y,
                                                bool, unsigned char *lines, const F &read) {
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
     fp64_fstat<L, N1, HALF>(v[0], a, b, blk * R + c, t);
}

// The row pass: one persistent CTA per SM.  A row block (RUN rows, one
// contiguous 128 L bytes of Y) takes about as long to load as to transform
// (2^18 points: 0.68 and 0.78 us per template alone), and CTAs that start
// together do the one and then the other (1.35-1.47 us against 1.05 as
// follows).  The blocks come in by bulk copies into
// split_row_bufs() buffers while the split_row_groups() thread groups of the
// CTA transform earlier ones in place, 16 warps of up to 128 registers (two
// lines per thread share the pass twiddles).
// CTA c's j-th block is block c + j*gridDim.x; group j % G transforms it in
// buffer j % NB, and once the group has read its last exchange its thread 0
// starts the copy of block j + NB into that buffer and notes it in issued[]
// (a group that got ahead of the buffer's previous user must not take that
// user's barrier phase for its own).  A block's copy depends on the block NB
// before it only, so every wait ends; all are bounded.  A thread whose wait
// gave up reports ERR_STAGE_TIMEOUT in *err and neither waits nor starts a copy
// again: it only keeps its group's barriers, and the groups whose blocks are
// then never copied give up in turn.  Before the CTA leaves, every copy that was
// started is waited for.
// (FP64: the same block and buffer bytes, four rows, one line per thread.)
template <int L> __host__ __device__ constexpr int split_row_threads() { return L / 2; }   // of a group
// Half as many buffers again as 512 threads' groups fit the shared memory; with
// short lines the split form gives one of the spare ones to a fifth group (96
// registers): 2^17 points 0.561 -> 0.547 us per template, 2^16 0.341 -> 0.326.
template <class V, int L> __host__ __device__ constexpr int split_row_cta() { return sizeof(V) == 8 && L == 256 ? 640 : 512; }
template <class V, int L> __host__ __device__ constexpr int split_row_groups() { return split_row_cta<V, L>() / split_row_threads<L>(); }
template <int L> __host__ __device__ constexpr int split_row_bufs() {
     return L >= 1024 ? 1 : 512 / split_row_threads<L>() * 3 / 2;
}
template <class V, int L> __host__ __device__ constexpr size_t split_row_smem() {
     return split_row_bufs<L>() * (SplitLine<V, L, true>::BYTES + sizeof(uint64_t) + sizeof(int));
}

// makes this thread's earlier accesses to shared memory (and those it has
// observed) precede the bulk copies it starts next
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async;" ::: "memory"); }

template <class A, int L, int N1, bool HALF>
__global__ void __launch_bounds__(split_row_cta<typename A::V, L>(), 1) k_row(const __grid_constant__ A a) {
     using V = typename A::V;
     extern __shared__ __align__(128) unsigned char smem_raw[];
     constexpr int GT = split_row_threads<L>(), G = split_row_groups<V, L>(), NB = split_row_bufs<L>();
     constexpr unsigned BYTES = SplitLine<V, L, true>::BYTES, COPY = 2 * sizeof(V) * L * run_of<V>;
     static_assert(COPY <= BYTES, "a row block must fit in its exchange buffer");
     constexpr int BPT = N1 / run_of<V>;   // blocks per template
     uint64_t *full = reinterpret_cast<uint64_t *>(smem_raw + NB * BYTES);
     volatile int *issued = reinterpret_cast<volatile int *>(full + NB);   // the block a buffer's copy brings
     const int n = (a.nt * BPT - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;   // this CTA's blocks
     auto copy = [&](int j) {
          const size_t item = blockIdx.x + (size_t)j * gridDim.x;
          mbar_expect_tx(&full[j % NB], COPY);
          bulk_load(smem_raw + (j % NB) * BYTES, a.y + item * (COPY / sizeof(V)), COPY, &full[j % NB]);
          __threadfence_block();
          issued[j % NB] = j;
     };
     if (threadIdx.x == 0) {
          for (int i = 0; i < NB; i++) {
               mbar_init(&full[i], 1);
               issued[i] = -1;
          }
          mbar_fence_init();
          for (int j = 0; j < NB && j < n; j++) copy(j);
     }
     __syncthreads();
     const int g = threadIdx.x / GT, tid = threadIdx.x % GT;
     bool ok = true;
     for (int j = g; j < n; j += G) {
          unsigned char *buf = smem_raw + (j % NB) * BYTES;
          if (ok) {
               int probes = 4 * a.probes;
               while (issued[j % NB] != j && --probes > 0) {}
               __threadfence_block();
               ok = probes > 0 && mbar_wait(&full[j % NB], (unsigned)(j / NB) & 1u, a.probes);
          }
          const int item = (int)blockIdx.x + j * (int)gridDim.x;
          split_row_block<L, N1, HALF>(a, item / BPT, item % BPT, tid, g, reinterpret_cast<const V *>(buf), true, buf,
                                       [&] {
                                            group_sync<L / 2>(g);   // the group is done with the buffer
                                            if (tid == 0 && ok && j + NB < n) {
                                                 fence_proxy_async();
                                                 copy(j + NB);
                                            }
                                       });
     }
     if (!ok) atomicOr(a.err, ERR_STAGE_TIMEOUT);
     if (__syncthreads_or(!ok) && threadIdx.x == 0)
          for (int i = 0; i < NB; i++)
               if (issued[i] >= 0) mbar_wait(&full[i], (unsigned)(issued[i] / NB) & 1u);
}

// ------------------------------------------------------------------ fused pass order
//
// k_spinpass runs the column pass and the row pass of nt templates (FP32, two
// arrays, N1 = N2 = L) as one launch of persistent CTAs (as many as are
// resident at once).  C = R = L/RUN blocks per template and pass; the
// items are handed out by tickets (ctl[0]) in the order
//   col(0) .. col(D-1), then for b = 0 .. nt-D-1: col(b+D), row(b),
//   then row(nt-D) .. row(nt-1)
// (col(b) = the C column blocks of template b, row(b) its R row blocks), so
// that a template's rows follow its columns by about D templates while its
// spectra Y are still in L2.  A CTA takes its next ticket while it works on
// the current item.  When a CTA starts the item after a column block of
// template b, its thread 0 publishes that block (device-scope fence, then
// ctl[2+b] += 1): the fence overlaps the new item instead of holding the
// CTA.  A row block of template b waits until ctl[2+b] == C (bounded: on
// time-out ERR_ORDER_TIMEOUT goes to *err and the block goes on).
// No deadlock: a CTA publishes before it waits, and waits only for items of
// smaller tickets; the waiting CTA whose current ticket is smallest depends
// on items that are finished, current in CTAs that wait on nothing, or next
// in CTAs whose current item has a smaller ticket and so is not waiting.
// ctl is zeroed (memset) before each launch.
constexpr unsigned ERR_ORDER_TIMEOUT = 8u;

struct SpinOrder {
     unsigned *ctl;   // [0] tickets, [1] unused, [2 + b] column blocks done of template b
     unsigned *err;
     int nt, C, R, D;
     int limit;       // probes of a row block's wait
};

__host__ __device__ __forceinline__ void spin_item(const SpinOrder &o, unsigned k, int &b, int &blk, bool &row) {
     const unsigned C = (unsigned)o.C, R = (unsigned)o.R, D = (unsigned)o.D;
     const unsigned head = D * C;
     if (k < head) {
          row = false;
          b = (int)(k / C);
          blk = (int)(k % C);
          return;
     }
     k -= head;
     const unsigned mid = (unsigned)(o.nt - o.D) * (C + R);
     if (k < mid) {
          const unsigned g = k / (C + R), r = k % (C + R);
          row = r >= C;
          b = (int)(row ? g : g + D);
          blk = (int)(row ? r - C : r);
          return;
     }
     k -= mid;
     row = true;
     b = (int)((unsigned)(o.nt - o.D) + k / R);
     blk = (int)(k % R);
}

__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned *p) {
     unsigned v;
     asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
     return v;
}

// Waits until *p >= target, giving up after `limit` probes; returns false
// when it gave up.
__device__ __forceinline__ bool wait_count(const unsigned *p, unsigned target, int limit) {
     for (int it = 0; it < limit; it++) {
          if (ld_acquire_gpu(p) >= target) return true;
          __nanosleep(64);
     }
     return ld_acquire_gpu(p) >= target;
}

// (Y is written and read within the launch: the row blocks read it with
// __ldcg, past L1.)
template <int L, bool HALF>
__global__ void __launch_bounds__(split_row_threads<L>(), 512 / split_row_threads<L>())
k_spinpass(const __grid_constant__ SplitCol col, const __grid_constant__ SplitRow row_, const __grid_constant__ SpinOrder o) {
     extern __shared__ __align__(128) unsigned char smem_raw[];
     __shared__ unsigned s_tk[2];
     const unsigned total = (unsigned)o.nt * (unsigned)(o.C + o.R);
     if (threadIdx.x == 0) s_tk[0] = atomicAdd(&o.ctl[0], 1u);
     __syncthreads();
     int pend = -1;         // template of the column block finished last, not yet published
     for (int it = 0;; it++) {
          const unsigned k = s_tk[it & 1];
          if (threadIdx.x == 0) {
               if (pend >= 0) {
                    __threadfence();
                    atomicAdd(&o.ctl[2 + pend], 1u);
               }
               if (k < total) s_tk[(it + 1) & 1] = atomicAdd(&o.ctl[0], 1u);
          }
          pend = -1;
          if (k >= total) break;
          int b, blk;
          bool row;
          spin_item(o, k, b, blk, row);
          if (!row) {
               const int line = threadIdx.x / (L / 8), t = threadIdx.x % (L / 8);
               unsigned char *s = smem_raw + line * SplitLine<float2, L, false>::BYTES;
               // RUN columns, two in turn for each of the CTA's RUN/2 thread groups
               split_col_line<L, L, 2, 1>(col, b, blk * RUN + 2 * line, t, line, s);
               group_sync<L / 8>(line);
               split_col_line<L, L, 2, 1>(col, b, blk * RUN + 2 * line + 1, t, line, s);
               pend = b;
          } else {
               if (threadIdx.x == 0) {
                    if (!wait_count(&o.ctl[2 + b], (unsigned)o.C, o.limit)) atomicOr(o.err, ERR_ORDER_TIMEOUT);
               }
               __syncthreads();
               split_row_block<L, L, HALF>(row_, b, blk, threadIdx.x, 0,
                                                row_.y + ((size_t)b * L + (size_t)blk * RUN) * (2 * L), false, smem_raw, [] {});
          }
          __syncthreads();   // the item's shared memory is free; the next ticket is visible
     }
}

}  // namespace tdf
