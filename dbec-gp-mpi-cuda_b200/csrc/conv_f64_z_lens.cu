// conv_f64_z_lens.cu -- FP64 inverse z pass (conv_lens.cuh).
#include "conv_lens.cuh"

template gpe_status zinv_lens<double>(gpe_solver *, size_t);
