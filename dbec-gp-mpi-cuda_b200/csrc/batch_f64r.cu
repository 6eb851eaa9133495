// batch_f64r.cu -- batched step of FP64 real-time groups.
#include "batch_step.cuh"

extern template gpe_status BatchConv<double>::run(const Group &, cudaStream_t, cudaEvent_t *);
template gpe_status batch_step<double, true>(const Group &, cudaStream_t, long long *, cudaEvent_t *);
