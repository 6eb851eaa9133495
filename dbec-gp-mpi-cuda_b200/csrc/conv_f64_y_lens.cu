// conv_f64_y_lens.cu -- FP64 y passes on the lengths compiled for one solve only.
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
template gpe_status yfft_lens<double>(gpe_solver *, bool, unsigned, size_t);
