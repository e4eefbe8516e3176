// passes_x_f64_b.cu -- batched x passes of double fields.
#include "kernels.cuh"

namespace pmgpu {

template <> RxBatchKernel rx_batch_kernel<double>(bool inverse) {
  return inverse ? k_rxinv_batch<double, 3> : k_rxfwd_batch<double, 3>;
}

int upload_cs_x_f64_b(const void *t32, const void *t64) { return upload_cs_local(t32, t64); }

}  // namespace pmgpu
