// passes_x_f32_b.cu -- batched x passes of float fields.
#include "kernels.cuh"

namespace pmgpu {

template <> RxBatchKernel rx_batch_kernel<float>(bool inverse) {
  return inverse ? k_rxinv_batch<float2, 3> : k_rxfwd_batch<float2, 3>;
}

int upload_cs_x_f32_b(const void *t32, const void *t64) { return upload_cs_local(t32, t64); }

}  // namespace pmgpu
