// apply_f64.cu -- the fused-wave FP64 apply (apply_fused.cuh).
#include "apply_fused.cuh"

namespace symeig {
template int64_t fused_layers_per_pass<double>(int64_t, int64_t);
template size_t fused_table_bytes<double>(int64_t, int64_t);
template size_t fused_state_bytes<double>(int64_t);
template cudaError_t fused_pass<double, double>(double*, int64_t, int64_t, const double*, int64_t, const int32_t*,
                                                const ApplyPass&, void*, int*, cudaStream_t, cudaEvent_t, cudaEvent_t, int);
template cudaError_t fused_host_segmented<double>(double*, int64_t, const double*, const ApplyPass&, void*, int*,
                                                  cudaStream_t, const HostStream&);
}  // namespace symeig
