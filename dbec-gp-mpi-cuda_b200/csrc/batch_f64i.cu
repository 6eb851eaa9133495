// batch_f64i.cu -- batched step of FP64 imaginary-time groups.
#include "batch_step.cuh"

template gpe_status BatchConv<double>::run(const Group &, cudaStream_t, cudaEvent_t *);
template gpe_status batch_step<double, false>(const Group &, cudaStream_t, long long *, cudaEvent_t *);
