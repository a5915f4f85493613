// apply_f32.cu -- the fused-wave FP32 apply (apply_fused.cuh).
#include "apply_fused.cuh"

namespace symeig {
template int64_t fused_layers_per_pass<float>(int64_t, int64_t);
template size_t fused_table_bytes<float>(int64_t, int64_t);
template size_t fused_state_bytes<float>(int64_t);
template cudaError_t fused_pass<float, float>(float*, int64_t, int64_t, const float*, int64_t, const int32_t*,
                                              const ApplyPass&, void*, int*, cudaStream_t, cudaEvent_t, cudaEvent_t, int);
template cudaError_t fused_pass<double, float>(float*, int64_t, int64_t, const double*, int64_t, const int32_t*,
                                               const ApplyPass&, void*, int*, cudaStream_t, cudaEvent_t, cudaEvent_t, int);
template cudaError_t fused_host_segmented<float>(float*, int64_t, const float*, const ApplyPass&, void*, int*,
                                                 cudaStream_t, const HostStream&);
}  // namespace symeig
