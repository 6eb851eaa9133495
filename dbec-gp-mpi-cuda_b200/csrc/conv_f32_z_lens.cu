// conv_f32_z_lens.cu -- mixed-precision inverse z pass on the lengths compiled for one solve only.
#include "impl.cuh"

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
template gpe_status zinv_lens<float>(gpe_solver *, size_t);
