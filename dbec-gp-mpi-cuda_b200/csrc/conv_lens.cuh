// conv_lens.cuh -- the passes of the dipolar convolution on the lengths compiled
// for one solve only (instantiated in conv_*_lens.cu, one translation unit per
// pass and real type).
#pragma once

#include "impl.cuh"

template <class R> gpe_status yfft_lens(gpe_solver *s, bool inv, unsigned grid, size_t sm) {
   constexpr int L = LenCols<R>::L;
   return with_len_xy(s->d.ny, [&](auto nc) -> gpe_status {
      constexpr int N = decltype(nc)::value;
      if constexpr (N > 0) {
         auto go = [&](auto k) -> gpe_status {
            return launch_pdl(k, grid, len_threads<R>(N, L), sm, s, s->tm_spec_y, s->d, (const cpx<R> *) s->twy, s->err);
         };
         return inv ? go(k_yfft_n<R, true, L, N>) : go(k_yfft_n<R, false, L, N>);
      } else {
         return fail(GPE_ERR_STATE, "no compile-time y pass for this length");
      }
   });
}

template <class R> gpe_status xconv_lens(gpe_solver *s, unsigned grid, size_t sm) {
   constexpr int L = LenCols<R>::L;
   return with_len_xy(s->d.nx, [&](auto nc) -> gpe_status {
      constexpr int N = decltype(nc)::value;
      if constexpr (N > 0) {
         return launch_pdl(k_xconv_n<R, L, N>, grid, len_threads<R>(N, L), sm, s, s->tm_spec_x, s->tm_udd, s->d,
                           (const cpx<R> *) s->twx, s->state, s->err);
      } else {
         return fail(GPE_ERR_STATE, "no compile-time x pass for this length");
      }
   });
}

template <class R> gpe_status zinv_lens(gpe_solver *s, size_t sm) {
   return with_len_z(s->d.nz / 2, [&](auto nc) -> gpe_status {
      constexpr int H = decltype(nc)::value;
      if constexpr (H > 0 && (sizeof(R) == 8 || H % 2 == 0)) {  // mixed precision: nz divisible by 4
         return launch_pdl(k_zinv_n<R, kLenRows, H>, blocks_for(s->d.nxy, kLenRows), len_threads<R>(H, kLenRows), sm, s,
                           (const cpx<R> *) s->spec, (R *) s->phi, s->d, (const cpx<R> *) s->twz, s->err);
      } else {
         return fail(GPE_ERR_STATE, "no compile-time z pass for this length");
      }
   });
}

template <class R, bool CPLX> gpe_status zfwd_lens(gpe_solver *s, size_t sm) {
   return with_len_z(s->d.nz / 2, [&](auto nc) -> gpe_status {
      constexpr int H = decltype(nc)::value;
      if constexpr (H > 0 && (sizeof(R) == 8 || H % 2 == 0)) {  // mixed precision: nz divisible by 4
         using P = typename Tr<R, CPLX>::P;
         return launch_pdl(k_zfwd_n<R, CPLX, kLenRows, H>, blocks_for(s->d.nxy, kLenRows), len_threads<R>(H, kLenRows), sm,
                           s, (const P *) s->psi, (cpx<R> *) s->spec, s->d, (const cpx<R> *) s->twz, s->err);
      } else {
         return fail(GPE_ERR_STATE, "no compile-time z pass for this length");
      }
   });
}
