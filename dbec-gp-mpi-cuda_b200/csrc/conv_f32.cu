// conv_f32.cu -- convolution passes of mixed-precision handles.
#include "impl.cuh"

template gpe_status Conv<float>::rest(gpe_solver *);
