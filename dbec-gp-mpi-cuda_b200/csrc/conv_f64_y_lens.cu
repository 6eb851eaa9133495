// conv_f64_y_lens.cu -- FP64 y passes (conv_lens.cuh).
#include "conv_lens.cuh"

template gpe_status yfft_lens<double>(gpe_solver *, bool, unsigned, size_t);
