// conv_f32_zf_lens.cu -- Mixed-precision forward z pass (conv_lens.cuh).
#include "conv_lens.cuh"

template gpe_status zfwd_lens<float, false>(gpe_solver *, size_t);
template gpe_status zfwd_lens<float, true>(gpe_solver *, size_t);
