// impl_f64i.cu -- operators of FP64 imaginary-time handles.
#include "impl.cuh"

extern template gpe_status Conv<double>::rest(gpe_solver *);
template struct Ops<double, false>;
