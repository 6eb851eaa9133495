// conv_f32_x_lens.cu -- Mixed-precision x convolution (conv_lens.cuh).
#include "conv_lens.cuh"

template gpe_status xconv_lens<float>(gpe_solver *, unsigned, size_t);
