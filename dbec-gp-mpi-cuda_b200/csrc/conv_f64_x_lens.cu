// conv_f64_x_lens.cu -- FP64 x convolution (conv_lens.cuh).
#include "conv_lens.cuh"

template gpe_status xconv_lens<double>(gpe_solver *, unsigned, size_t);
