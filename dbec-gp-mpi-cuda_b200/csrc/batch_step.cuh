// batch_step.cuh -- the launches of a batched step.
#pragma once

#include "batch_group.h"

template <class K, class... A>
gpe_status launch(const Group &G, K kern, unsigned grid, unsigned block, size_t smem, cudaStream_t st, A... args) {
   if (grid == 0) return GPE_OK;
   BCK(G.roomy.allow((const void *) kern, smem));
   kern<<<grid, block, smem, st>>>(args...);
   BCK(cudaGetLastError());
   return GPE_OK;
}

// The convolution passes that do not see psi (y, x and inverse z FFTs).
template <class R> struct BatchConv {
   // mixed precision: phi's boundary planes are stored by the inverse z pass
   // (batch of 64: a pass of 13 us less); an FP64 batch step keeps its
   // documented launch per pass
   static constexpr bool kFold = std::is_same<R, float>::value;
   // runs f(lens, points per thread) as compile-time constants
   template <class F> static gpe_status with_fft(const BatchGeom &A, int q, F f) {
      auto go = [&](auto lens) -> gpe_status {
         if constexpr (std::is_same<R, double>::value)
            if (A.ppt[q] == 8) return f(lens, std::integral_constant<int, 8>());
         return f(lens, std::integral_constant<int, 16>());
      };
      return A.lens[q] ? go(std::true_type()) : go(std::false_type());
   }
   template <class F> static gpe_status with_L(int L, F f) {
      if constexpr (std::is_same<R, float>::value)  // a tile row is 128 bytes at most
         if (L >= 16) return f(std::integral_constant<int, 16>());
      if (L >= 8) return f(std::integral_constant<int, 8>());
      if (L == 4) return f(std::integral_constant<int, 4>());
      return f(std::integral_constant<int, 2>());
   }
   static gpe_status run(const Group &G, cudaStream_t st, cudaEvent_t *ev);
};

template <class R> gpe_status BatchConv<R>::run(const Group &G, cudaStream_t st, cudaEvent_t *ev) {
   const BatchGeom &A = G.geo;
   const BatchDesc *tab = G.dtab;
   auto S = [&](int q) { return (const unsigned *) (G.dwork + G.off[q]); };
   auto T = [&](int q) { return (unsigned) A.tiles[q]; };
   constexpr int ZL = 8;
   auto mark = [&](int q) -> gpe_status {
      if (ev) BCK(cudaEventRecord(ev[q], st));
      return GPE_OK;
   };
   BCKS(with_L(G.Ly, [&](auto lc) {
      return with_fft(A, kPYfft, [&](auto nc, auto pc) {
         return launch(G, kb_yfft<R, false, decltype(pc)::value, decltype(lc)::value, decltype(nc)::value>, T(kPYfft), A.threads[kPYfft],
                       A.smem[kPYfft], st, tab, S(kPYfft));
      });
   }));
   BCKS(mark(kPYfft));
   BCKS(with_L(G.Lx, [&](auto lc) {
      return with_fft(A, kPXconv, [&](auto nc, auto pc) {
         return launch(G, kb_xconv<R, decltype(pc)::value, decltype(lc)::value, decltype(nc)::value>, T(kPXconv), A.threads[kPXconv],
                       A.smem[kPXconv], st, tab, S(kPXconv));
      });
   }));
   BCKS(mark(kPXconv));
   BCKS(with_L(G.Ly, [&](auto lc) {
      return with_fft(A, kPYinv, [&](auto nc, auto pc) {
         return launch(G, kb_yfft<R, true, decltype(pc)::value, decltype(lc)::value, decltype(nc)::value>, T(kPYinv), A.threads[kPYinv],
                       A.smem[kPYinv], st, tab, S(kPYinv));
      });
   }));
   BCKS(mark(kPYinv));
   BCKS(with_fft(A, kPZinv, [&](auto nc, auto pc) {
      return launch(G, kb_zinv<R, decltype(pc)::value, ZL, kFold, decltype(nc)::value>, T(kPZinv), A.threads[kPZinv],
                    A.smem[kPZinv], st, tab, S(kPZinv));
   }));
   BCKS(mark(kPZinv));
   if (!kFold) BCKS(launch(G, kb_phifix<R>, T(kPPhifix), A.threads[kPPhifix], 0, st, tab, S(kPPhifix)));
   BCKS(mark(kPPhifix));
   return GPE_OK;
}

// The passes of one batch step of group G, on stream st.
template <class R, bool CPLX> struct BatchStep {
   using C = cpx<R>;
   static constexpr bool kFold = BatchConv<R>::kFold;
   template <class F> static gpe_status with_mseg(int m, F f) {
      if constexpr (std::is_same<R, float>::value && !CPLX)
         if (m > 16) return f(std::integral_constant<int, 32>());
      if constexpr (!(std::is_same<R, double>::value && CPLX))  // 16-byte elements: 8-point segments
         if (m > 8) return f(std::integral_constant<int, 16>());
      return f(std::integral_constant<int, 8>());
   }

   // ev (may be null): an event recorded after every pass, index = pass
   static gpe_status run(const Group &G, cudaStream_t st, long long *kernels, cudaEvent_t *ev = nullptr) {
      const BatchGeom &A = G.geo;
      const BatchDesc *tab = G.dtab;
      auto S = [&](int q) { return (const unsigned *) (G.dwork + G.off[q]); };
      auto T = [&](int q) { return (unsigned) A.tiles[q]; };
      constexpr int ZL = 8;
      auto mark = [&](int q) -> gpe_status {
         if (ev) BCK(cudaEventRecord(ev[q], st));
         return GPE_OK;
      };
      BCKS(BatchConv<R>::with_fft(A, kPZfwd, [&](auto nc, auto pc) {
         return launch(G, kb_zfwd<R, CPLX, decltype(pc)::value, ZL, decltype(nc)::value>, T(kPZfwd), A.threads[kPZfwd],
                       A.smem[kPZfwd], st, tab, S(kPZfwd));
      }));
      BCKS(mark(kPZfwd));
      BCKS(BatchConv<R>::run(G, st, ev));
      BCKS(with_mseg(A.mseg[0], [&](auto mc) {
         constexpr int M = decltype(mc)::value;
         return launch(G, kb_sweep_xy<R, CPLX, 0, true, M, 2>, (unsigned) G.sweep_grid[0], A.threads[kPXsweep],
                       G.sweep_smem[0], st, tab, (const SweepTile *) G.dtile[0], (int) A.tiles[kPXsweep], A.stage[0], A.xch[0], A.tabs[0], G.nbuf[0]);
      }));
      BCKS(mark(kPXsweep));
      BCKS(with_mseg(A.mseg[1], [&](auto mc) {
         constexpr int M = decltype(mc)::value;
         return launch(G, kb_sweep_xy<R, CPLX, 1, false, M, 2>, (unsigned) G.sweep_grid[1], A.threads[kPYsweep],
                       G.sweep_smem[1], st, tab, (const SweepTile *) G.dtile[1], (int) A.tiles[kPYsweep], A.stage[1], A.xch[1], A.tabs[1], G.nbuf[1]);
      }));
      BCKS(mark(kPYsweep));
      BCKS(with_mseg(A.mseg[2], [&](auto mc) {
         constexpr int M = decltype(mc)::value;
         constexpr int MOM = CPLX ? 0 : 1;
         return launch(G, kb_sweep_z<R, CPLX, MOM, M, 2>, (unsigned) G.sweep_grid[2], A.threads[kPZsweep],
                       G.sweep_smem[2], st, tab, (const SweepTile *) G.dtile[2], (int) A.tiles[kPZsweep], A.stage[2], A.xch[2], A.tabs[2], G.nbuf[2],
                       A.part);
      }));
      BCKS(mark(kPZsweep));
      if (!CPLX) BCKS(launch(G, kb_norm_final, T(kPNorm), A.threads[kPNorm], 0, st, tab, S(kPNorm)));
      BCKS(mark(kPNorm));
      *kernels += (CPLX ? 9 : 10) - (kFold ? 1 : 0);
      return GPE_OK;
   }
};

template <class R, bool CPLX>
gpe_status batch_step(const Group &G, cudaStream_t st, long long *kernels, cudaEvent_t *ev) {
   return BatchStep<R, CPLX>::run(G, st, kernels, ev);
}
