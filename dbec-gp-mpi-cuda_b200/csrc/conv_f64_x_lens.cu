// conv_f64_x_lens.cu -- FP64 x convolution on the lengths compiled for one solve only.
#include "impl.cuh"

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
template gpe_status xconv_lens<double>(gpe_solver *, unsigned, size_t);
