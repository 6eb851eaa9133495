// impl_f32i.cu -- operators of mixed-precision imaginary-time handles.
#include "impl.cuh"

extern template gpe_status Conv<float>::rest(gpe_solver *);
template struct Ops<float, false>;
