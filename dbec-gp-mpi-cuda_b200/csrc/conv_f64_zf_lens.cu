// conv_f64_zf_lens.cu -- FP64 forward z pass (conv_lens.cuh).
#include "conv_lens.cuh"

template gpe_status zfwd_lens<double, false>(gpe_solver *, size_t);
template gpe_status zfwd_lens<double, true>(gpe_solver *, size_t);
