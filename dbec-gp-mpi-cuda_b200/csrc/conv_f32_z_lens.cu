// conv_f32_z_lens.cu -- Mixed-precision inverse z pass (conv_lens.cuh).
#include "conv_lens.cuh"

template gpe_status zinv_lens<float>(gpe_solver *, size_t);
