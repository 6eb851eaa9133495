// conv_f64.cu -- convolution passes of FP64 handles.
#include "impl.cuh"

template gpe_status Conv<double>::rest(gpe_solver *);
