// impl_f64r.cu -- operators of FP64 real-time handles.
#include "impl.cuh"

extern template gpe_status Conv<double>::rest(gpe_solver *);
template struct Ops<double, true>;
