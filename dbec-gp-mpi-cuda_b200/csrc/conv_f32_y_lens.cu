// conv_f32_y_lens.cu -- Mixed-precision y passes (conv_lens.cuh).
#include "conv_lens.cuh"

template gpe_status yfft_lens<float>(gpe_solver *, bool, unsigned, size_t);
