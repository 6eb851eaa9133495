// sweep_kernels.cuh -- Crank-Nicolson Thomas sweeps along x, y and z
// (calclux/calcluy/calcluz_kernel, imag3d-mpicuda.cu:1802-1942,
// real3d-mpicuda.cu:1902-2040) on whole lines staged in shared memory.
//
// A CTA owns TW lines.  The lines are brought in by one TMA tensor load (x
// and y sweeps: box of TW z-columns by the whole line) or by one bulk copy
// per row (z sweep), so every HBM access is a full 128-byte row segment and
// no transpose is needed.  Each line is cut into P segments of exactly m
// points, one thread per (line, segment); the two first-order recurrences of
// the Thomas algorithm
//    beta[i-1] = gamma[i] (A beta[i] - c_i),      i = n-2 .. 1
//    psi'[i+1] = alpha[i] psi'[i] + beta[i],      i = 0 .. n-3
// run locally from a zero carry-in, and the true values follow from the
// carries by the exact decomposition value = local + prefix_product * carry,
// with the prefix products of (gamma_i A) and alpha_i precomputed per axis
// (tables M and N).  The result equals the sequential recurrence up to
// rounding.
//
// Segments are aligned at the top of the line: segment p owns the recurrence
// indices lo .. lo + m - 1, lo = p m - skip with skip = P m - (n - 2), so the
// top one ends at n - 3 and the bottom one starts skip rows below the line.
// Those rows are zero and the tables hold zero coefficients there (so beta
// and psi' are exactly zero below index 1): no index of the unrolled loops
// needs a bound check.
//
// Carries: segment p maps the value entering at its top to beta[lo] by the
// affine map x -> b_p + a_p x with a_p = M at its bottom.  |a_p| is the decay
// of the recurrence over one segment (alpha^m, alpha about dt / (4 dx^2):
// 1e-13 for dt = 0.1 dx^2 and m = 8), so a carry from D segments away is
// scaled by a product of D such factors.  The host picks the smallest D for
// which that product stays below 2^-64 (FP64) or 2^-40 (FP32), 2^-11 and
// 2^-16 of the type's rounding unit (D = 1 or 2 for the usual time steps, up
// to P for large ones), and a thread composes the maps of the D segments
// beyond its own from a shared table of the b_p.  The scan over all segments
// that this replaces (shuffles in the warp, then a chain over the warps) cost
// about as many instructions as the recurrences.
#pragma once

#include <type_traits>

#include "kernels.cuh"
#include "step_kernels.cuh"
#include "tma.cuh"

namespace gpe {

// Segment tables of one axis, indexed by p m + q (recurrence index i = lo + q
// of segment p): FP64 for the FP64 sweeps, once-rounded FP32 for the FP32 ones.
struct SegTab {
   const void *ga;  // gamma[i + 1]
   const void *ma;  // pairs (M[i], alpha[i])
   const void *nn;  // N[i + 1]
   double2 A;
   int n, m, P, D, skip;
};

// Bytes of the zero rows below a tile of TW lines (kept a multiple of the 128
// bytes a TMA destination is aligned to).
__host__ __device__ __forceinline__ uint32_t sweep_pad(int skip, int TW, int esz) {
   return (uint32_t) ((skip * TW * esz + 127) & ~127);
}

template <class R, bool CPLX> struct SegOps {
   using P = typename Tr<R, CPLX>::P;
   // coefficient entry: from global memory (read-only path) or staged in
   // shared memory
   template <bool STAB> __device__ __forceinline__ static P ld(const P *t) {
      if constexpr (STAB) return *t;
      else return __ldg(t);
   }
   // 16 bytes of a table: V entries
   static constexpr int V = 16 / (int) sizeof(P);
   template <bool STAB> __device__ __forceinline__ static void ldv(const P *t, P (&o)[V]) {
      if constexpr (sizeof(P) == 4) {
         const float4 v = STAB ? *(const float4 *) t : __ldg((const float4 *) t);
         o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
      } else if constexpr (std::is_same<P, float2>::value) {
         const float4 v = STAB ? *(const float4 *) t : __ldg((const float4 *) t);
         o[0] = make_float2(v.x, v.y); o[1] = make_float2(v.z, v.w);
      } else if constexpr (sizeof(P) == 8) {
         const double2 v = STAB ? *(const double2 *) t : __ldg((const double2 *) t);
         o[0] = v.x; o[1] = v.y;
      } else {
         o[0] = ld<STAB>(t);
      }
   }
   // One backward Thomas step of the Crank-Nicolson system.  With the
   // coefficients of gencoef, minusA = -A and A0r = 1 + 2A in both modes
   // (imag: A = -c/2 real; real: A = -i c/2), so the right-hand side
   //    r = minusA psi[i+1] + A0r psi[i] - A psi[i-1] = psi[i] + A t,
   //    t = 2 psi[i] - psi[i+1] - psi[i-1],
   // and gamma (A beta - r) = gamma (A (beta - t) - psi[i]).  `a` is A's
   // real (imag mode) or imaginary (real mode) part.
   //
   // FP32 real time: gamma = -1 / (A0 + A alpha) is -1 plus a small complex
   // number (about i c), and a once-rounded FP32 gamma is off by up to half
   // an FP32 ulp of 1 at every index, the same error at every step: the
   // solve is then not unitary and the norm and mu drift linearly (1.7e-5
   // and 5.7e-5 after 200 steps of a 32x30x40 test, the error of the whole
   // mixed path; rounding alpha, A, psi, phi or the calcnu phase factor to
   // FP32 instead changes mu by at most 2e-8 there, measured with the FP64
   // oracle).  So the FP32 table holds gamma + 1, whose rounding error is
   // that of the small part.  The small products are summed before u (and, in
   // fma_, before c): one rounding at psi's magnitude per component where a
   // chain of two multiply-adds has two.  After 100 mixed real-time steps, over
   // 48 draws of spacing, time step and g, rms against FP64: psi 2.2e-6 ->
   // 1.6e-6, mu 6.8e-7 -> 5.0e-7, for 352 -> 358 us a step at 256^3.
   __device__ static P back_step(P b, P w2, P w1, P w0, P g, R a) {
      if constexpr (CPLX) {
         const R tx = fma((R) 2, w1.x, -w2.x) - w0.x, ty = fma((R) 2, w1.y, -w2.y) - w0.y;
         const R dx = b.x - tx, dy = b.y - ty;
         const R ux = fma(-a, dy, -w1.x), uy = fma(a, dx, -w1.y);
         P r;
         if constexpr (std::is_same<R, float>::value) {  // g = gamma + 1
            r.x = fma(g.x, ux, -g.y * uy) - ux;
            r.y = fma(g.x, uy, g.y * ux) - uy;
         } else {
            r.x = fma(g.x, ux, -g.y * uy);
            r.y = fma(g.x, uy, g.y * ux);
         }
         return r;
      } else {
         const R t = fma((R) 2, w1, -w2) - w0;
         return g * fma(a, b - t, -w1);
      }
   }
   __device__ static P fma_(P a, P b, P c) {  // a * b + c
      if constexpr (CPLX) {
         P r;
         if constexpr (std::is_same<R, float>::value) {
            r.x = c.x + fma(a.x, b.x, -a.y * b.y);
            r.y = c.y + fma(a.x, b.y, a.y * b.x);
         } else {
            r.x = fma(a.x, b.x, c.x);
            r.x = fma(-a.y, b.y, r.x);
            r.y = fma(a.x, b.y, c.y);
            r.y = fma(a.y, b.x, r.y);
         }
         return r;
      } else {
         return fma(a, b, c);
      }
   }
};

// Own points of a segment as they are (the y and z sweeps): w[q] = lp[q es].
struct NoXf {
   static constexpr bool kNu = false;
};

// Segmented Thomas sweep of one line in shared memory (element i at
// line[i es], rows -skip .. -1 present), by all threads of the CTA: thread p
// of the line owns segment p of M points, threads with p >= tb.P only take
// part in the barriers.  xch points at this line's column of an exchange
// buffer of 2 P rows of xs elements.  The swept line is written back in
// place.  ROW: es == 1 and 16-byte aligned rows, accessed in pairs.  STAB:
// the tables are in shared memory.
//
// xf may transform the points first (the x sweep's calcnu): a thread
// transforms its own M points into registers, publishes the two lowest (the
// ones the segment below also reads) in the line, and the top thread
// transforms the two points above the last segment itself.
//
// SIMP 1: *simp receives this thread's share of sum_i |psi'_i|^2 with the
// Simpson weights, 4 at odd i and 2 at even i inside the line by parity (lo is
// even).  SIMP 2:
// with the weights w1[i] into *simp and w2[i] into *simp2 (both arrays have
// skip entries before index 0).
template <class R, bool CPLX, int M, bool ROW, bool STAB, int SIMP, class XF>
__device__ __forceinline__ void seg_sweep(typename Tr<R, CPLX>::P *line, int es_, int p, const SegTab &tb,
                                          typename Tr<R, CPLX>::P *xch, int xs, const XF &xf,
                                          const double *w1t = nullptr, const double *w2t = nullptr,
                                          double *simp = nullptr, double *simp2 = nullptr) {
   using Op = SegOps<R, CPLX>;
   using P = typename Tr<R, CPLX>::P;
   constexpr int V = Op::V;
   const int es = ROW ? 1 : es_;
   const int NP = tb.P;
   const bool act = p < NP, top = p == NP - 1;
   const int lo = p * M - tb.skip;
   const R a = CPLX ? (R) tb.A.y : (R) tb.A.x;
   P *lp = line + lo * es;
   const P *ga = (const P *) tb.ga + p * M, *ma = (const P *) tb.ma + 2 * p * M, *nn = (const P *) tb.nn + p * M;
   P *xb = xch, *xv = xch + NP * xs;

   P w[M];
   P t2 = zero_of<P>(), t1 = zero_of<P>();  // the two points above the segment
   if (act) {
      if (p == 0) {  // zero rows below the line (only this thread reads them)
         for (int q = 0; q < tb.skip; q++) lp[q * es] = zero_of<P>();
         if constexpr (XF::kNu)
            for (int q = 0; q < tb.skip; q++) xf.zero_row(q - tb.skip);
      }
      if constexpr (XF::kNu) {
         xf.template own<M>(lp, lo, w);
         if (top) {
            P tt[2];
            xf.template own<2>(lp + M * es, lo + M, tt);
            t1 = tt[0];
            t2 = tt[1];
         }
         lp[0] = w[0];
         lp[es] = w[1];
      } else if constexpr (ROW) {
#pragma unroll
         for (int q = 0; q < M; q += 2) ld2(lp + q, w[q], w[q + 1]);
         ld2(lp + M, t1, t2);
      } else {
#pragma unroll
         for (int q = 0; q < M; q++) w[q] = lp[q * es];
         t1 = lp[M * es];
         t2 = lp[(M + 1) * es];
      }
   }
   if constexpr (XF::kNu) {
      __syncthreads();
      if (act && !top) {
         t1 = lp[M * es];
         t2 = lp[(M + 1) * es];
      }
   }

   // ---- backward local recurrence: bt[q] = beta~[lo + q]
   P bt[M];
   if (act) {
      P b = top ? t2 : zero_of<P>();  // beta[n-2] = psi[n-1] is exact
#pragma unroll
      for (int q0 = M - V; q0 >= 0; q0 -= V) {
         P g[V];
         Op::template ldv<STAB>(ga + q0, g);
#pragma unroll
         for (int j = V - 1; j >= 0; j--) {
            const int q = q0 + j;
            b = Op::back_step(b, q + 2 < M ? w[q + 2 < M ? q + 2 : 0] : (q + 1 < M ? t1 : t2),
                              q + 1 < M ? w[q + 1 < M ? q + 1 : 0] : t1, w[q], g[j], a);
            bt[q] = b;
         }
      }
      xb[p * xs] = b;
   }
   __syncthreads();  // also: every read of the line is complete before it is rewritten
   P v = zero_of<P>();
   if (act) {
      // ---- beta entering at the top of this segment
      P bin = zero_of<P>();
      int s = min(p + tb.D, NP - 1);
      if (s > p) bin = xb[s * xs];
      for (s--; s > p; s--) bin = Op::fma_(Op::template ld<STAB>((const P *) tb.ma + 2 * s * M), bin, xb[s * xs]);
      // ---- forward local recurrence: bt[q] becomes psi'~[lo + q + 1]
#pragma unroll
      for (int q0 = 0; q0 < M; q0 += (V > 1 ? V / 2 : 1)) {
         constexpr int G = V > 1 ? V / 2 : 1;  // (M, alpha) pairs per 16 bytes
         P c[2 * G];
         if constexpr (V > 1) {
            P cc[V];
            Op::template ldv<STAB>(ma + 2 * q0, cc);
#pragma unroll
            for (int j = 0; j < V; j++) c[j] = cc[j];
         } else {
            c[0] = Op::template ld<STAB>(ma + 2 * q0);
            c[1] = Op::template ld<STAB>(ma + 2 * q0 + 1);
         }
#pragma unroll
         for (int j = 0; j < G; j++) {
            const P beta = Op::fma_(c[2 * j], bin, bt[q0 + j]);
            v = Op::fma_(c[2 * j + 1], v, beta);
            bt[q0 + j] = v;
         }
      }
      xv[p * xs] = v;
   }
   __syncthreads();
   double acc = 0., acc2 = 0., acc_o = 0., acc_e = 0.;
   if (act) {
      // ---- psi' entering at the bottom of this segment (zero for p = 0)
      P fin = zero_of<P>();
      int s = max(p - tb.D, 0);
      if (s < p) fin = xv[s * xs];
      for (s++; s < p; s++) fin = Op::fma_(Op::template ld<STAB>((const P *) tb.nn + s * M + M - 1), fin, xv[s * xs]);
#pragma unroll
      for (int q0 = 0; q0 < M; q0 += V) {
         P g[V];
         Op::template ldv<STAB>(nn + q0, g);
#pragma unroll
         for (int j = 0; j < V; j++) {
            const int q = q0 + j;
            bt[q] = Op::fma_(g[j], fin, bt[q]);
            if constexpr (SIMP == 1) {
               const double f = (double) dens2(bt[q]);
               if (q & 1) acc_e += f;  // index lo + q + 1 even
               else acc_o += f;
            } else if constexpr (SIMP == 2) {
               const double f = (double) dens2(bt[q]);
               acc += w1t[lo + q + 1] * f;
               acc2 += w2t[lo + q + 1] * f;
            }
         }
      }
      if constexpr (ROW) {
         lp[1] = bt[0];
#pragma unroll
         for (int q = 1; q + 1 < M; q += 2) st2(lp + q + 1, bt[q], bt[q + 1]);
         lp[M] = bt[M - 1];
      } else {
#pragma unroll
         for (int q = 0; q < M; q++) lp[(q + 1) * es] = bt[q];
      }
      if (p == 0) line[0] = zero_of<P>();
      if (top) line[(tb.n - 1) * es] = zero_of<P>();
   }
   if constexpr (SIMP == 1) {
      *simp = fma(4., acc_o, 2. * acc_e);
      // the end correction of an even line: the weights of points n-2 and n-3
      // are 3 and 3.75 where the interior weights give 2 and 4
      if (top && !(tb.n & 1)) *simp += (double) dens2(bt[M - 1]) - 0.25 * (double) dens2(bt[M - 2]);
   }
   if constexpr (SIMP == 2) {
      *simp = acc;
      *simp2 = acc2;
   }
}

// The same for the run-time segment length of the table (8, 16 or, up to
// MMAX, 32 points).
template <class R, bool CPLX, int MMAX, bool ROW, bool STAB, int SIMP, class XF>
__device__ __forceinline__ void seg_sweep_any(typename Tr<R, CPLX>::P *line, int es, int p, const SegTab &tb,
                                              typename Tr<R, CPLX>::P *xch, int xs, const XF &xf,
                                              const double *w1t = nullptr, const double *w2t = nullptr,
                                              double *simp = nullptr, double *simp2 = nullptr) {
   if constexpr (MMAX >= 32)
      if (tb.m == 32) return seg_sweep<R, CPLX, 32, ROW, STAB, SIMP>(line, es, p, tb, xch, xs, xf, w1t, w2t, simp, simp2);
   if constexpr (MMAX >= 16)
      if (tb.m == 16) return seg_sweep<R, CPLX, 16, ROW, STAB, SIMP>(line, es, p, tb, xch, xs, xf, w1t, w2t, simp, simp2);
   seg_sweep<R, CPLX, 8, ROW, STAB, SIMP>(line, es, p, tb, xch, xs, xf, w1t, w2t, simp, simp2);
}

// (cos t, -sin t) on |t| <= 1/32: sin through t^7, cos through t^6 (omitted
// terms below 3e-18 relative to sin and 3e-17 to cos).
__device__ __forceinline__ double2 expi_series7(double t) {
   constexpr double s3 = 1. / 6, s5 = s3 / 20, s7 = s5 / 42, c2 = 1. / 2, c4 = c2 / 12, c6 = c4 / 30;
   const double t2 = t * t;
   double sq = fma(-s7, t2, s5);
   sq = fma(sq, t2, -s3);
   double cq = fma(-c6, t2, c4);
   cq = fma(cq, t2, -c2);
   return make_double2(fma(cq, t2, 1.), -fma(sq * t2, t, t));
}

// exp(-i t) = (cos t, -sin t) for the nonlinear part of the real-time phase,
// which is small in practice: Maclaurin series on |t| <= 1/32 (through t^7
// for sin and t^6 for cos; the first omitted terms are below 3e-18 relative
// to sin and 3e-17 to cos) and on |t| <= 0.25 (through t^11 and t^12; below
// 3e-18), the library sincos beyond.  The short series is the common case:
// with it the 256^3 FP64 real-time step (dt = 4e-4, g = 200) measured 0.817
// -> 0.815 ms on B200.
__device__ __forceinline__ double2 expi_small(double t) {
   if (fabs(t) > 0.25) {
      double sn, cs;
      sincos(-t, &sn, &cs);
      return make_double2(cs, sn);
   }
   if (fabs(t) <= 0.03125) return expi_series7(t);
   constexpr double s3 = 1. / 6, s5 = s3 / 20, s7 = s5 / 42, s9 = s7 / 72, s11 = s9 / 110;
   constexpr double c2 = 1. / 2, c4 = c2 / 12, c6 = c4 / 30, c8 = c6 / 56, c10 = c8 / 90, c12 = c10 / 132;
   const double t2 = t * t;
   double sp = fma(-s11, t2, s9);
   sp = fma(sp, t2, -s7);
   sp = fma(sp, t2, s5);
   sp = fma(sp, t2, -s3);
   const double sn = fma(sp * t2, t, t);
   double cp = fma(c12, t2, -c10);
   cp = fma(cp, t2, c8);
   cp = fma(cp, t2, -c6);
   cp = fma(cp, t2, c4);
   cp = fma(cp, t2, -c2);
   const double cs = fma(cp, t2, 1.);
   return make_double2(cs, -sn);
}

// calcnu of the x sweep (calcnu_kernel, imag3d-mpicuda.cu:1759,
// real3d-mpicuda.cu:1856) on the points of one line column: the pending 1/norm
// first, then the trap and nonlinear factors.  V is a sum over the axes, so
// its factor is a product of per-axis ones: `fix` holds the part of the two
// coordinates the column fixes, xt the table along the line.
//
// own<M>() transforms a thread's segment straight into registers with the
// short series that holds for small nonlinear exponents (the usual case), all
// points unrolled; a thread that met a larger exponent redoes its points one
// by one in place (one(), which picks the series or the library function per
// point) and reloads them.  Transforming the tile in a pass of its own took
// 82 instructions per FP64 point in imaginary time, mostly indexing and the
// second trip through shared memory.

// (cos t, -sin t) in FP32 on |t| <= 256: t is reduced by the nearest multiple
// of pi / 2 in two steps (Cody and Waite), then Maclaurin series on |r| <= pi/4
// (sine through r^9, cosine through r^10; omitted terms below 3e-9).
__device__ __forceinline__ float2 expi_f32(float t) {
   constexpr double pio2 = 1.57079632679489661923;
   constexpr float hi = (float) pio2, lo = (float) (pio2 - (double) hi), inv = (float) (1. / pio2);
   constexpr float s3 = (float) (1. / 6), s5 = (float) (1. / 120), s7 = (float) (1. / 5040), s9 = (float) (1. / 362880),
                   c2 = 0.5f, c4 = (float) (1. / 24), c6 = (float) (1. / 720), c8 = (float) (1. / 40320),
                   c10 = (float) (1. / 3628800);
   const float km = fmaf(t, inv, 12582912.f);  // 1.5 2^23: the sum's low bits are the rounded multiple
   const int q = __float_as_int(km);
   const float k = km - 12582912.f;
   const float r = fmaf(k, -lo, fmaf(k, -hi, t)), r2 = r * r;
   float sq = fmaf(s9, r2, -s7);
   sq = fmaf(sq, r2, s5);
   sq = fmaf(sq, r2, -s3);
   const float sn = fmaf(sq * r2, r, r);
   float cq = fmaf(-c10, r2, c8);
   cq = fmaf(cq, r2, -c6);
   cq = fmaf(cq, r2, c4);
   cq = fmaf(cq, r2, -c2);
   const float cs = fmaf(cq, r2, 1.f);
   const float c = q & 1 ? sn : cs, s = q & 1 ? cs : sn;  // up to sign
   return make_float2((q + 1) & 2 ? -c : c, q & 2 ? s : -s);
}

// XS: the table along the line is in shared memory (always in FP64).
template <class R, bool CPLX, bool XS> struct NuXf {
   using P = typename Tr<R, CPLX>::P;
   using T = typename std::conditional<CPLX && std::is_same<R, double>::value, double2, R>::type;
   static constexpr bool kNu = true;
   R *ph;        // phi of this column, row i at ph[i es]
   int es;
   // along the line: exp(-dt V_x) in imaginary time, the phase exp(-i dt V_x)
   // in FP64 real time, x^2 in FP32 real time
   const T *xt;
   T fix;        // the other two factors; FP32 real time: unused
   R scale, dtg, dtgd;      // 1/norm, dt g, dt gd / N
   R ca, to, tz, hp, dt;    // FP32 real time: V = hp ((ca x^2 + to) + tz)

   __device__ __forceinline__ static T ldx(const T *p) {
      if constexpr (XS) return *p;
      else return __ldg(p);
   }
   __device__ __forceinline__ void zero_row(int i) const { ph[i * es] = (R) 0; }

   __device__ __forceinline__ R expo(P p, R f) const {  // nonlinear exponent
      return fma(dens2(p), dtg, f * dtgd);
   }
   // FP32 real time: the whole exponent.  It stays one phase: FP32 factors
   // per axis would each round cos and sin near 1, the same error at every
   // step.
   __device__ __forceinline__ float expo32(float2 p, float f, float x2) const {
      const float sv = __fadd_rn(__fadd_rn(__fmul_rn(ca, x2), to), tz);
      return fmaf(dt, __fmul_rn(hp, sv), fmaf(dens2(p), dtg, f * dtgd));
   }

   __device__ __forceinline__ P one(P v, int i) const {
      if constexpr (std::is_same<R, double>::value && !CPLX) {
         const double p = v * scale;
         return p * ((xt[i] * fix) * exp_small(-expo(p, ph[i * es])));
      } else if constexpr (std::is_same<R, double>::value) {
         return cmul(v, cmul(cmul(xt[i], fix), expi_small(expo(v, ph[i * es]))));
      } else if constexpr (!CPLX) {
         const float p = v * scale;
         return p * ((xt[i] * fix) * expf(-expo(p, ph[i * es])));
      } else {
         float sn, cs;
         sincosf(-expo32(v, ph[i * es], xt[i]), &sn, &cs);
         return cmul(v, make_float2(cs, sn));
      }
   }

   template <int M> __device__ __forceinline__ void own(P *lp, int lo, P (&w)[M]) const {
      const R *f = ph + lo * es;
      const T *x = xt + lo;
      bool big = false;
#pragma unroll
      for (int q = 0; q < M; q++) {
         if constexpr (std::is_same<R, double>::value && !CPLX) {
            const double p = lp[q * es] * scale, t = expo(p, f[q * es]);
            big |= !(fabs(t) <= 0.125);
            w[q] = p * ((x[q] * fix) * exp_series10(-t));
         } else if constexpr (std::is_same<R, double>::value) {
            const double2 p = lp[q * es];
            const double t = expo(p, f[q * es]);
            big |= !(fabs(t) <= 0.03125);
            w[q] = cmul(p, cmul(cmul(x[q], fix), expi_series7(t)));
         } else if constexpr (!CPLX) {
            const float p = lp[q * es] * scale;
            w[q] = p * ((ldx(x + q) * fix) * expf(-expo(p, f[q * es])));
         } else {
            const float2 p = lp[q * es];
            const float t = expo32(p, f[q * es], ldx(x + q));
            big |= !(fabsf(t) <= 256.f);
            w[q] = cmul(p, expi_f32(t));
         }
      }
      if (big) {
#pragma unroll 1
         for (int q = 0; q < M; q++) lp[q * es] = one(lp[q * es], lo + q);
#pragma unroll
         for (int q = 0; q < M; q++) w[q] = lp[q * es];
      }
   }
};

// The functor of tile column c of an x sweep tile covering z columns
// [z0, z0 + TW) of plane y = other; pcol is phi's column in the tile, xtab the
// table along the line staged in shared memory, `skip` zero entries before
// index 0 (XS; else the FP32 tables are read through L1).
template <class R, bool CPLX, bool XS>
__device__ __forceinline__ NuXf<R, CPLX, XS> nu_xf(R *pcol, int TW, int other, int z0, int c, const Dims &d,
                                                   const Trap &trap, const LinPhase &lin, const void *xtab, int skip,
                                                   double g, double gd, double dt, double scale) {
   const int k = min(z0 + c, d.nz - 1);  // columns past nz are zero fill, never stored
   NuXf<R, CPLX, XS> f;
   using T = typename NuXf<R, CPLX, XS>::T;
   f.ph = pcol;
   f.es = TW;
   f.scale = (R) scale;
   f.dtg = (R) (dt * g);
   f.dtgd = (R) (dt * gd / (double) d.npts);
   if constexpr (std::is_same<R, float>::value && CPLX) {
      f.xt = XS ? (const T *) xtab + skip : trap.x2f;
      f.fix = 0.f;
      f.ca = (float) trap.vg2;
      f.to = __fmul_rn((float) trap.vn2, trap.y2f[other]);
      f.tz = __fmul_rn((float) trap.vl2, trap.z2f[k]);
      f.hp = (float) trap.hp;
      f.dt = (float) dt;
   } else {
      const T ey = __ldg((const T *) lin.ey + other), ez = __ldg((const T *) lin.ez + k);
      if constexpr (CPLX) f.fix = cmul(ey, ez);
      else f.fix = ey * ez;
      f.xt = XS ? (const T *) xtab + skip : (const T *) lin.ex;
      f.ca = f.to = f.tz = f.hp = f.dt = (R) 0;
   }
   return f;
}

// ---------------------------------------------------------------------------
// Persistent pipelined CTAs.  A CTA walks the tiles t = blockIdx.x,
// blockIdx.x + gridDim.x, ... through S shared-memory stages: while it sweeps
// tile i, the TMA engine already loads tile i+1 into the next stage and
// stores tile i-1 from the previous one.  Thread 0 issues every copy; before
// refilling a stage it waits until the bulk store that last read the stage
// has finished reading (all but the newest S-2 store groups: wait_stage_free).
//
// Resident CTAs of 256 threads per SM the sweep kernels are compiled for
// (register budget); the host never launches more per SM.
__host__ __device__ constexpr int sweep_ctas(bool fp32, bool cplx, int m) {
   if (fp32) return m == 32 ? 2 : (cplx && m == 16 ? 3 : 4);
   return !cplx && m == 8 ? 3 : 2;
}

// CTAs of `bytes` of dynamic shared memory that an SM holds: each also takes the
// kernel's static bytes (`fixed`: at most 128 for these kernels) and the 1 KB the
// system reserves.  A persistent grid of more CTAs than that runs the surplus
// after the others have finished: 16 complex FP64 64^3 solves in a batch, six
// CTAs launched where five fit, x sweep 111 us, z 48; as many as fit 86 and 35.
constexpr size_t kSmSmem = 228 * 1024, kCtaReserved = 1024, kSweepFixed = 128;
inline int smem_ctas(size_t bytes, size_t fixed) {
   return (int) (kSmSmem / ((bytes + fixed + kCtaReserved + 127) & ~(size_t) 127));
}

// Shared-memory layout of one pipeline stage of an x or y sweep tile: zero
// rows below the tile, the tile, and with calcnu the same for phi.
struct XyStage {
   uint32_t psi, phi, bytes;  // offsets of row 0 of psi and phi, size of the stage
};
template <class R, bool CPLX, bool NU>
__host__ __device__ __forceinline__ XyStage xy_stage(int rows, int TW, int skip) {
   constexpr int esz = (int) sizeof(R) * (CPLX ? 2 : 1);
   XyStage g;
   g.psi = sweep_pad(skip, TW, esz);
   g.phi = g.bytes = g.psi + (uint32_t) ((rows * TW * esz + 127) & ~127);
   if (NU) {
      g.phi += sweep_pad(skip, TW, (int) sizeof(R));
      g.bytes = g.phi + (uint32_t) ((rows * TW * (int) sizeof(R) + 127) & ~127);
   }
   return g;
}

// calcnu's per-x table staged in shared memory (FP64: the tiles leave little
// L1 for it), with `skip` zero entries before index 0.
template <bool CPLX> __device__ __forceinline__ void stage_xtab(double *xtab, const void *ex, int n, int skip) {
   constexpr int E = CPLX ? 2 : 1;
   const double *src = (const double *) ex;
   for (int e = threadIdx.x; e < E * (n + skip); e += blockDim.x) xtab[e] = e < E * skip ? 0. : src[e - E * skip];
}

// x or y sweep.  Tile: TW consecutive z columns of one y (x sweep) or one x
// (y sweep) plane, the whole line along the swept axis, brought in by TMA.
// With NU the x sweep first applies the pending 1/norm and calcnu to the tile
// (needs phi).  Bound by issue, not bytes: two CTAs of 128 registers (four of 64
// in FP32) issue on a third (FP32 half) of the cycles.  256^3 on B200, with a
// scan over the segments -> with carries from D segments, us (bytes at 6.65
// TB/s): x FP64 complex 209 -> 167 (101), real 144 -> 90 (60), FP32 real 88
// -> 54 (30), complex 98 now (50); y FP64 complex 127 -> 106 (81), real 70 -> 52 (40),
// FP32 real 51 -> 30 (20).
template <class R, bool CPLX, int AXIS, bool NU, int MSEG, int S, int TWC>
__global__ void __launch_bounds__(256, sweep_ctas(sizeof(R) == 4, CPLX, MSEG)) k_sweep_xy(const __grid_constant__ CUtensorMap tm_psi,
                                                     const __grid_constant__ CUtensorMap tm_phi, Dims d, SegTab tb,
                                                     Trap trap, LinPhase lin, double g, double gd, double dt,
                                                     const State *__restrict__ st, int tw_arg, int boxn, int nbox,
                                                     uint32_t *err) {
   pdl_trigger();
   using P = typename Tr<R, CPLX>::P;
   const int TW = TWC > 0 ? TWC : tw_arg;
   extern __shared__ __align__(16) unsigned char smem_raw[];
   __shared__ __align__(8) uint64_t full[S];
   const int n = tb.n;
   const int rows = boxn * nbox;  // rows staged (>= n)
   constexpr int E = CPLX ? 2 : 1;
   const XyStage lay = xy_stage<R, CPLX, NU>(rows, TW, tb.skip);
   const uint32_t tx = (uint32_t) (rows * TW * sizeof(P)) + (NU ? (uint32_t) (rows * TW * sizeof(R)) : 0u);
   // layout: S stages | exchange buffer | calcnu table  (TMA targets 128-byte aligned)
   unsigned char *base = (unsigned char *) (((uintptr_t) smem_raw + 127) & ~(uintptr_t) 127);
   P *xch = (P *) (base + S * lay.bytes);
   double *xtab = (double *) (xch + 2 * tb.P * TW);
   const int nzb = (d.nz + TW - 1) / TW;
   const int ntiles = (AXIS == 0 ? d.ny : d.nx) * nzb;
   auto copy_tile = [&](int t, int q, bool load) {
      const int other = t / nzb, z0 = (t - other * nzb) * TW;
      P *tile = (P *) (base + q * lay.bytes + lay.psi);
      R *ptile = (R *) (base + q * lay.bytes + lay.phi);
      if (load) mbar_arrive_expect_tx(&full[q], tx);
      for (int b = 0; b < nbox; b++) {
         const int a0 = b * boxn;
         if (load) {
            if (AXIS == 0) tma_load_3d(tile + a0 * TW, &tm_psi, E * z0, other, a0, &full[q]);
            else tma_load_3d(tile + a0 * TW, &tm_psi, E * z0, a0, other, &full[q]);
            if (NU) {
               if (AXIS == 0) tma_load_3d(ptile + a0 * TW, &tm_phi, z0, other, a0, &full[q]);
               else tma_load_3d(ptile + a0 * TW, &tm_phi, z0, a0, other, &full[q]);
            }
         } else {
            if (AXIS == 0) tma_store_3d(&tm_psi, E * z0, other, a0, tile + a0 * TW);
            else tma_store_3d(&tm_psi, E * z0, a0, other, tile + a0 * TW);
         }
      }
      if (!load) bulk_commit();
   };
   if constexpr (NU && std::is_same<R, double>::value) stage_xtab<CPLX>(xtab, lin.ex, n, tb.skip);
   if (threadIdx.x == 0) {
      for (int q = 0; q < S; q++) mbar_init(&full[q], 1);
      fence_mbar_init();
   }
   pdl_wait();  // the tables above do not depend on the previous kernel
   if (threadIdx.x == 0 && (int) blockIdx.x < ntiles) copy_tile(blockIdx.x, 0, true);
   __syncthreads();
   const double scale = NU ? st->scale : 1.;
   const int lg = __ffs(TW) - 1;  // TW is a power of two
   const int c = threadIdx.x & (TW - 1), p = threadIdx.x >> lg;
   int i = 0;
   for (int t = blockIdx.x; t < ntiles; t += gridDim.x, i++) {
      const int q = i % S;
      if (threadIdx.x == 0 && t + (int) gridDim.x < ntiles) {
         wait_stage_free<S>();
         copy_tile(t + gridDim.x, (i + 1) % S, true);
      }
      // a timed-out copy makes the whole CTA leave together
      if (__syncthreads_or(!mbar_wait(&full[q], (i / S) & 1, err))) break;
      P *col = (P *) (base + q * lay.bytes + lay.psi) + c;
      if constexpr (NU) {
         static_assert(AXIS == 0, "calcnu is fused into the x sweep only");
         const int other = t / nzb, z0 = (t - other * nzb) * TW;
         seg_sweep<R, CPLX, MSEG, false, false, 0>(
             col, TW, p, tb, xch + c, TW,
             nu_xf<R, CPLX, std::is_same<R, double>::value>((R *) (base + q * lay.bytes + lay.phi) + c, TW, other, z0, c,
                                                            d, trap, lin, xtab, tb.skip, g, gd, dt, scale));
      } else {
         seg_sweep<R, CPLX, MSEG, false, false, 0>(col, TW, p, tb, xch + c, TW, NoXf());
      }
      fence_proxy_async();
      __syncthreads();
      if (threadIdx.x == 0) copy_tile(t, q, false);
   }
   if (threadIdx.x == 0) bulk_wait_all();
}

// Entries before element 0 of a staged z row (room for the zero entries,
// rounded so that element 0 stays 16-byte aligned) and the row stride: an odd
// number of 16-byte units, so that the rows of a warp fall on different banks.
__host__ __device__ __forceinline__ int zrow_pad(int skip, int esz) {
   const int u = 16 / esz;
   return (skip + u - 1) / u * u;
}
__host__ __device__ __forceinline__ int zrow_stride(int nz, int skip, int esz) {
   const int u = 16 / esz;
   const int units = (nz + zrow_pad(skip, esz) + u - 1) / u;
   return (units | 1) * u;
}

// What the z sweep leaves besides psi.  MOM 1 (imaginary time): per tile the
// sum over its rows of w_x w_y S_z |psi'|^2 (tile, the norm's partials).  MOM
// 2: per row S_z |psi'|^2 and S_z z^2 |psi'|^2 (row partials of calcrms).
struct ZOut {
   const double *wz, *wz2;  // Simpson weights along z (MOM 2)
   double hz3;
   double *tile, *rowA, *rowB;
};

// The z sweep of one staged tile of TR rows (nr of them inside the grid;
// `rows` is element 0 of the first, LS the row stride) starting at grid row
// row0; ends with the tile written back in shared memory and a CTA barrier
// (the caller then stores it).
template <class R, bool CPLX, int MOM, int MSEG, bool STAB, bool ANY>
__device__ __forceinline__ void zsweep_tile(typename Tr<R, CPLX>::P *rows, int nr, int TR, int LS, int c, int p,
                                            const SegTab &tbs, typename Tr<R, CPLX>::P *xch, double *part,
                                            double *part2, const Dims &d, const ZOut &o, long long row0, int tile) {
   using P = typename Tr<R, CPLX>::P;
   constexpr bool SIMP = MOM >= 1;
   if (nr < TR) {  // rows beyond the grid are zero so their sweep stays finite
      for (int e = threadIdx.x; e < (TR - nr) * tbs.n; e += blockDim.x)
         rows[(nr + e / tbs.n) * LS + e % tbs.n] = zero_of<P>();
      __syncthreads();
   }
   double my = 0., my2 = 0.;
   if constexpr (ANY)
      seg_sweep_any<R, CPLX, MSEG, true, STAB, MOM>(rows + c * LS, 1, p, tbs, xch + c, TR, NoXf(), o.wz, o.wz2, &my, &my2);
   else
      seg_sweep<R, CPLX, MSEG, true, STAB, MOM>(rows + c * LS, 1, p, tbs, xch + c, TR, NoXf(), o.wz, o.wz2, &my, &my2);
   if (SIMP && p < tbs.P) part[p * TR + c] = my;
   if (MOM == 2 && p < tbs.P) part2[p * TR + c] = my2;
   fence_proxy_async();
   __syncthreads();
   // the rows' sums on the last warp, so that warp 0 (whose lanes issue the
   // tile's store and the next load) goes on at once: 32 / TR lanes per row
   const int ln = (int) threadIdx.x - ((int) blockDim.x - 32);
   if (SIMP && ln >= 0) {
      const int rr = ln % TR;
      double sum = 0., sum2 = 0.;
      if (rr < nr)
         for (int pp = ln / TR; pp < tbs.P; pp += 32 / TR) {
            sum += part[pp * TR + rr];
            if (MOM == 2) sum2 += part2[pp * TR + rr];
         }
      for (int q = TR; q < 32; q <<= 1) {
         sum += __shfl_xor_sync(0xffffffffu, sum, q);
         if (MOM == 2) sum2 += __shfl_xor_sync(0xffffffffu, sum2, q);
      }
      if (MOM == 2 && ln < nr) {
         o.rowA[row0 + rr] = sum * o.hz3;
         o.rowB[row0 + rr] = sum2 * o.hz3;
      }
      if (MOM == 1) {
         if (ln < nr) {
            const int row = (int) row0 + rr, i = row / d.ny, j = row - i * d.ny;
            sum *= o.hz3 * simp_w(i, d.nx) * simp_w(j, d.ny);
         } else {
            sum = 0.;
         }
         for (int q = 16; q; q >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, q);
         if (ln == 0) o.tile[tile] = sum;
      }
   }
}

// FP64: the coefficient tables staged in shared memory once per CTA, the
// shared rows leaving little L1 for them (z sweep 129 -> 128 us real, 94 -> 93
// us imaginary time at 256^3; FP32 measured slower with it).  4 P m entries.
template <bool CPLX> __device__ __forceinline__ SegTab stage_segtab(double *tabs, const SegTab &tb) {
   const int ne = tb.P * tb.m * (CPLX ? 2 : 1);
   SegTab o = tb;
   for (int e = threadIdx.x; e < ne; e += blockDim.x) {
      tabs[e] = ((const double *) tb.ga)[e];
      tabs[ne + e] = ((const double *) tb.ma)[e];
      tabs[2 * ne + e] = ((const double *) tb.ma)[ne + e];
      tabs[3 * ne + e] = ((const double *) tb.nn)[e];
   }
   o.ga = tabs;
   o.ma = tabs + ne;
   o.nn = tabs + 3 * ne;
   return o;
}

// z sweep.  Tile: TR consecutive (x, y) rows, each copied by one bulk copy to
// a padded shared row (zrow_pad, stride LS elements).  MOM 1 also yields the
// norm of the step (simpint, diffint.cu:106): the last CTA to finish adds the
// tile partials and sets the state (hx, hy; out_norm may be null), which was a
// launch of its own.  MOM 2 yields the row partials of calcrms, so an rms
// sample after the step needs no extra pass over psi.  Bound as the y sweep,
// with the Simpson sums on top; 256^3 on B200, us (bytes at 6.65 TB/s): FP64
// complex 131 -> 113 (81), real with the norm 89 + 10 -> 63 (40), FP32 real 62 +
// 10 -> 39 (20).
template <class R, bool CPLX, int MOM, int MSEG, int S, int TWC>
__global__ void __launch_bounds__(256, sweep_ctas(sizeof(R) == 4, CPLX, MSEG)) k_sweep_z(typename Tr<R, CPLX>::P *__restrict__ psi, Dims d, SegTab tb,
                                                    int tr_arg, int LS, ZOut out, double hx, double hy,
                                                    State *st, double *out_norm, uint32_t *err) {
   pdl_trigger();
   const int TR = TWC > 0 ? TWC : tr_arg;
   using P = typename Tr<R, CPLX>::P;
   extern __shared__ __align__(16) unsigned char smem_raw[];
   __shared__ __align__(8) uint64_t full[S];
   const int nz = d.nz;
   const uint32_t row_bytes = (uint32_t) (nz * sizeof(P));
   const uint32_t stage_bytes = ((uint32_t) (TR * LS * sizeof(P)) + 127u) & ~127u;
   const int pad = zrow_pad(tb.skip, (int) sizeof(P));
   // layout: S stages of rows | exchange buffer | Simpson partials | FP64 tables
   unsigned char *base = (unsigned char *) (((uintptr_t) smem_raw + 127) & ~(uintptr_t) 127);
   P *xch = (P *) (base + S * stage_bytes);
   double *part = (double *) ((unsigned char *) xch + ((2 * tb.P * TR * sizeof(P) + 15) & ~(size_t) 15));
   double *part2 = part + tb.P * TR;
   constexpr bool STAB = std::is_same<R, double>::value;
   double *tabs = part2 + tb.P * TR;
   SegTab tbs = tb;
   if constexpr (STAB) tbs = stage_segtab<CPLX>(tabs, tb);
   const int ntiles = (int) ((d.nxy + TR - 1) / TR);
   auto nrows = [&](int t) -> int {
      const long long r0 = (long long) t * TR;
      return (int) ((d.nxy - r0) < TR ? (d.nxy - r0) : TR);
   };
   // one bulk copy per row, issued by the lanes of warp 0 (one thread issuing
   // them kept the CTA waiting); every lane commits and waits for its own
   // store groups
   const int lane = threadIdx.x & 31;
   auto copy_tile = [&](int t, int q, bool load) {
      P *tile = (P *) (base + q * stage_bytes) + pad;
      const int nr = nrows(t);
      if (load && lane == 0) mbar_arrive_expect_tx(&full[q], row_bytes * nr);
      __syncwarp();
      for (int r = lane; r < nr; r += 32) {
         P *g = psi + ((long long) t * TR + r) * nz;
         if (load) bulk_load(tile + r * LS, g, row_bytes, &full[q]);
         else bulk_store(g, tile + r * LS, row_bytes);
      }
      if (!load) bulk_commit();
   };
   if (threadIdx.x == 0) {
      for (int q = 0; q < S; q++) mbar_init(&full[q], 1);
      fence_mbar_init();
   }
   __syncthreads();
   pdl_wait();  // the tables above do not depend on the previous kernel
   if (threadIdx.x < 32 && (int) blockIdx.x < ntiles) copy_tile(blockIdx.x, 0, true);
   const int c = threadIdx.x % TR, p = threadIdx.x / TR;
   int i = 0;
   for (int t = blockIdx.x; t < ntiles; t += gridDim.x, i++) {
      const int q = i % S;
      if (threadIdx.x < 32 && t + (int) gridDim.x < ntiles) {
         wait_stage_free<S>();
         copy_tile(t + gridDim.x, (i + 1) % S, true);
      }
      if (__syncthreads_or(!mbar_wait(&full[q], (i / S) & 1, err))) break;
      P *rows = (P *) (base + q * stage_bytes) + pad;
      zsweep_tile<R, CPLX, MOM, MSEG, STAB, false>(rows, nrows(t), TR, LS, c, p, tbs, xch, part, part2, d, out,
                                                   (long long) t * TR, t);
      if (threadIdx.x < 32) copy_tile(t, q, false);
   }
   if (threadIdx.x < 32) bulk_wait_all();
   if constexpr (MOM == 1) {
      __shared__ bool last;
      __shared__ double red[8];
      // the tile partials were written by this warp's lane 0
      if (threadIdx.x == blockDim.x - 32) {
         __threadfence();
         last = atomicAdd(&st->ticket, 1u) == gridDim.x - 1;
      }
      __syncthreads();
      if (!last) return;
      __threadfence();
      const double sum = sum_tiles(out.tile, ntiles, red);
      if (threadIdx.x == 0) {
         st->ticket = 0u;
         set_norm(st, sum, hx, hy, out_norm);
      }
   }
}

}  // namespace gpe
