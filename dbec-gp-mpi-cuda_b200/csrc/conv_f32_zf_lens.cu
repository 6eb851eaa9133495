// conv_f32_zf_lens.cu -- mixed-precision forward z pass on the lengths compiled for one solve only.
#include "impl.cuh"

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
template gpe_status zfwd_lens<float, false>(gpe_solver *, size_t);
template gpe_status zfwd_lens<float, true>(gpe_solver *, size_t);
