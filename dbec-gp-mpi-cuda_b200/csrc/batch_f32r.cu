// batch_f32r.cu -- batched step of mixed-precision real-time groups.
#include "batch_step.cuh"

extern template gpe_status BatchConv<float>::run(const Group &, cudaStream_t, cudaEvent_t *);
template gpe_status batch_step<float, true>(const Group &, cudaStream_t, long long *, cudaEvent_t *);
