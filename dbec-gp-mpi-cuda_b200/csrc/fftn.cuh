// fftn.cuh -- FFTs of compile-time length on lines in shared memory; fft.cuh
// transforms any other length.
//
// The transform is the one of fft.cuh (Stockham stages in the order of the
// same radix plan, the same roots of unity, L lines interleaved [j][L]), so
// both give the same values.  With the length, the line count and the CTA
// size known to the compiler every index is a constant offset from one base
// per butterfly: the run-time stages spent 100 warp instructions per point of
// a 256-point FP64 line of which 24 were FP64 arithmetic, the rest mostly
// integer indexing.  Three more things follow from the known plan:
//  - the roots of stage s lie in a table in the order the stage reads them
//    (stage_roots in solver.cu), one base address per butterfly;
//  - the first stage takes its points from a functor and the last one hands
//    them to a functor, so packing |psi|^2, the real-FFT merge and the final
//    row layout need no pass over shared memory of their own;
//  - a convolution keeps the points of the last forward stage in registers,
//    multiplies them and starts the inverse transform with the same radix on
//    them (conv_lines: the inverse runs the radices in reverse order).
#pragma once

#include <type_traits>
#include <utility>

#include "fft.cuh"

namespace gpe {

template <int... RS> struct Rads {};

// Points per thread of these passes, in both precisions.  FP64 threads hold 16
// points in 64 of their 128 registers; twice as many threads with 8 points and
// radices up to 8 measured slower at 256^3 (us: x 92 -> 78, z inverse 55.5 ->
// 50.6, z forward 60 -> 57).
constexpr int kLenPpt = 16;

// The lengths: a common set, compiled for one solve and for batches, with
// radices up to 16 in both precisions, and most other even lengths up to 400
// that factor into 2, 3 and 5, with half lengths for z, compiled for one solve
// only (above 256 a line is two boxes of 64-byte rows, so a multiple of 4).  The
// latter keep the radices of the run-time passes (16 in FP32, 8 in FP64), so a
// batch, which transforms them at run time, gives the same values bit for bit.
// The common set is the lines and half rows of sides of 48, 64, 96, 128, 256 and
// 512 points.  A batched kernel holds the code of all its lengths (a tile's
// instance is known at run time only), and in FP64 their 16 points a thread cost
// the run-time pass beside them half its warps (kb_fft_ctas), so the set is short.
// A whole step, their lengths at run time -> compiled, us: 128x96x80 FP64 70 ->
// 64, 90x100x72 FP64 complex 80 -> 72, 160x144x120 FP32 complex 120 -> 93.
#define GPE_LENS(X) X(24) X(32) X(48) X(64) X(96) X(128) X(256) X(512)
#define GPE_LENS_XY(X)                                                                                             \
   X(16) X(18) X(20) X(30) X(36) X(40) X(50) X(54) X(60) X(72) X(80) X(90) X(100) X(108) X(120) X(144) X(150) X(160) \
       X(162) X(180) X(192) X(200) X(216) X(240) X(250) X(288) X(300) X(320) X(324) X(360) X(384) X(400)
#define GPE_LENS_Z(X)                                                                                            \
   X(8) X(9) X(10) X(12) X(15) X(16) X(18) X(20) X(25) X(27) X(30) X(36) X(40) X(45) X(50) X(54) X(60) X(72) X(75) \
       X(80) X(81) X(90) X(100) X(108) X(120) X(125) X(135) X(144) X(150) X(160) X(162) X(180) X(192) X(200)
#define GPE_LEN_CASE(n) case n:
__host__ __device__ constexpr bool has_len(int n) {
   switch (n) {
      GPE_LENS(GPE_LEN_CASE) return true;
   default: return false;
   }
}
__host__ __device__ constexpr bool has_len_xy(int n) {
   switch (n) {
      GPE_LENS_XY(GPE_LEN_CASE) return true;
   default: return false;
   }
}
__host__ __device__ constexpr bool has_len_z(int h) {
   switch (h) {
      GPE_LENS_Z(GPE_LEN_CASE) return true;
   default: return false;
   }
}
#define GPE_LEN_CALL(n) \
   case n: return f(std::integral_constant<int, n>());
// runs f(std::integral_constant<int, n>) for a length of a set, with 0 for any
// other
template <class F> __host__ __device__ __forceinline__ auto with_len(int n, F f) {
   switch (n) {
      GPE_LENS(GPE_LEN_CALL)
   default: return f(std::integral_constant<int, 0>());
   }
}
template <class F> auto with_len_xy(int n, F f) {
   switch (n) {
      GPE_LENS_XY(GPE_LEN_CALL)
   default: return f(std::integral_constant<int, 0>());
   }
}
template <class F> auto with_len_z(int h, F f) {
   switch (h) {
      GPE_LENS_Z(GPE_LEN_CALL)
   default: return f(std::integral_constant<int, 0>());
   }
}

// Radix plan of a length, as make_radices lists it, and its reverse.
template <class R> __host__ __device__ constexpr int len_log(int n) { return has_len(n) || sizeof(R) == 4 ? 4 : 3; }
struct RadixList {
   int k;
   int r[kMaxStages];
};
constexpr RadixList radix_list(int n, int log2max) {
   RadixList l{};
   l.k = make_radices(n, log2max, l.r);
   return l;
}
template <int N, int LOG> struct RadixPlan {
   static constexpr RadixList l = radix_list(N, LOG);
   template <size_t... I> static Rads<l.r[I]...> up(std::index_sequence<I...>);
   template <size_t... I> static Rads<l.r[l.k - 1 - (int) I]...> down(std::index_sequence<I...>);
   using fwd = decltype(up(std::make_index_sequence<(size_t) l.k>()));
   using rev = decltype(down(std::make_index_sequence<(size_t) l.k>()));
};

// whether a convolution's inverse reads the same table of roots as its forward
template <class R, int N> __host__ __device__ constexpr bool palin_plan() {
   using PL = RadixPlan<N, len_log<R>(N)>;
   return std::is_same<typename PL::fwd, typename PL::rev>::value;
}

template <int RAD, int NB, int NT> struct StageRegs {
   static constexpr int U = (NB + NT - 1) / NT;  // butterflies per thread
};

// Reads and transforms this thread's butterflies of one stage (Ns = NS): v[u]
// holds butterfly b = tid + u NT of line b % L.  tw: this stage's roots,
// [t - 1][k].
template <int N, int L, int NT, int RAD, int NS, class C, bool INV, class LD, int U>
__device__ __forceinline__ void stage_read(C (&v)[U][RAD], const C *tw, const LD &ld) {
   constexpr int nr = N / RAD, nb = nr * L;
#pragma unroll
   for (int u = 0; u < U; u++) {
      const int b = threadIdx.x + u * NT;
      if ((int) threadIdx.x < NT && (nb % NT == 0 || b < nb)) {
         const int l = b % L, j = b / L;
#pragma unroll
         for (int t = 0; t < RAD; t++) v[u][t] = ld(l, j + t * nr);
         if constexpr (NS > 1) {
            const C *w0 = tw + j % NS;
#pragma unroll
            for (int t = 1; t < RAD; t++) {
               C w = w0[(t - 1) * NS];
               if (INV) w.y = -w.y;
               v[u][t] = cmul(v[u][t], w);
            }
         }
         dftr<RAD, C, INV>(v[u]);
      }
   }
}

// Hands the outputs of a stage to st(line, index, value).
template <int N, int L, int NT, int RAD, int NS, class C, class ST, int U>
__device__ __forceinline__ void stage_write(const C (&v)[U][RAD], const ST &st) {
   constexpr int nr = N / RAD, nb = nr * L;
#pragma unroll
   for (int u = 0; u < U; u++) {
      const int b = threadIdx.x + u * NT;
      if ((int) threadIdx.x < NT && (nb % NT == 0 || b < nb)) {
         const int l = b % L, j = b / L;
         const int o = (j / NS) * (NS * RAD) + j % NS;
#pragma unroll
         for (int t = 0; t < RAD; t++) st(l, o + t * NS, v[u][t]);
      }
   }
}

// The stages R0, RS... from Ns = NS on, in place on buf between the first
// stage's reads (ld) and the last one's writes (st).  tw: the roots of the
// first of them (the stage with Ns = 1 has none).  Every thread of the CTA
// calls it (NT of them work); ends without a barrier after the last writes.
template <int N, int L, int NT, class C, bool INV, int NS, int R0, int... RS, class LD, class ST>
__device__ __forceinline__ void stages(Rads<R0, RS...>, C *buf, const C *tw, const LD &ld, const ST &st) {
   constexpr int U = StageRegs<R0, N / R0 * L, NT>::U;
   {
      C v[U][R0];
      stage_read<N, L, NT, R0, NS, C, INV>(v, tw, ld);
      __syncthreads();
      if constexpr (sizeof...(RS) == 0) stage_write<N, L, NT, R0, NS, C>(v, st);
      else stage_write<N, L, NT, R0, NS, C>(v, [&](int l, int i, C x) { buf[i * L + l] = x; });
   }
   if constexpr (sizeof...(RS) > 0) {
      __syncthreads();
      stages<N, L, NT, C, INV, NS * R0>(Rads<RS...>(), buf, NS == 1 ? tw : tw + (R0 - 1) * NS,
                                        [&](int l, int i) { return buf[i * L + l]; }, st);
   }
}

// Transform of L lines of N points: point i of line l comes from ld(l, i) and
// goes to st(l, i, value).
template <int N, int L, int NT, class C, bool INV, class LD, class ST>
__device__ __forceinline__ void fft_lines(C *buf, const C *tw, const LD &ld, const ST &st) {
   using PL = RadixPlan<N, len_log<decltype(C::x)>(N)>;
   stages<N, L, NT, C, INV, 1>(typename PL::fwd(), buf, tw, ld, st);
}

// Forward transform, multiplication of point i of line l by mul(l, i), and
// inverse transform, in place on buf.  The last forward stage's outputs stay
// in registers: butterfly j ends on the points j + t N / RAD, exactly those
// the inverse's first stage (the same radix) starts from.
template <int N, int L, int NT, class C, int NS, int R0, int... RS, int I0, int... IS, class MUL>
__device__ __forceinline__ void conv_stages(Rads<R0, RS...>, Rads<I0, IS...> inv, C *buf, const C *tw, const C *twi,
                                            const MUL &mul) {
   constexpr int U = StageRegs<R0, N / R0 * L, NT>::U;
   auto ld = [&](int l, int i) { return buf[i * L + l]; };
   auto st = [&](int l, int i, C x) { buf[i * L + l] = x; };
   if constexpr (sizeof...(RS) > 0) {
      {
         C v[U][R0];
         stage_read<N, L, NT, R0, NS, C, false>(v, tw, ld);
         __syncthreads();
         stage_write<N, L, NT, R0, NS, C>(v, st);
      }
      __syncthreads();
      conv_stages<N, L, NT, C, NS * R0>(Rads<RS...>(), inv, buf, NS == 1 ? tw : tw + (R0 - 1) * NS, twi, mul);
   } else {
      static_assert(R0 == I0, "the inverse plan starts with the forward plan's last radix");
      {
         C v[U][R0];
         stage_read<N, L, NT, R0, NS, C, false>(v, tw, ld);
#pragma unroll
         for (int u = 0; u < U; u++) {
            const int b = threadIdx.x + u * NT;
            if ((int) threadIdx.x < NT && ((N / R0 * L) % NT == 0 || b < N / R0 * L)) {
               const int l = b % L, j = b / L;
#pragma unroll
               for (int t = 0; t < R0; t++) v[u][t] = scale_rn(v[u][t], mul(l, j + t * (N / R0)));
               dftr<R0, C, true>(v[u]);
            }
         }
         __syncthreads();
         stage_write<N, L, NT, R0, 1, C>(v, st);
      }
      if constexpr (sizeof...(IS) > 0) {
         __syncthreads();
         stages<N, L, NT, C, true, R0>(Rads<IS...>(), buf, twi, ld, st);
      }
   }
}
template <int N, int L, int NT, class C, class MUL>
__device__ __forceinline__ void conv_lines(C *buf, const C *tw, const C *twi, const MUL &mul) {
   using PL = RadixPlan<N, len_log<decltype(C::x)>(N)>;
   conv_stages<N, L, NT, C, 1>(typename PL::fwd(), typename PL::rev(), buf, tw, twi, mul);
}

}  // namespace gpe
