// impl_f32r.cu -- operators of mixed-precision real-time handles.
#include "impl.cuh"

extern template gpe_status Conv<float>::rest(gpe_solver *);
template struct Ops<float, true>;
