// batch_f32i.cu -- batched step of mixed-precision imaginary-time groups.
#include "batch_step.cuh"

template gpe_status BatchConv<float>::run(const Group &, cudaStream_t, cudaEvent_t *);
template gpe_status batch_step<float, false>(const Group &, cudaStream_t, long long *, cudaEvent_t *);
