// passes_x_f32_3.cu -- x passes of float fields of 3 components (two rows a vector).
#include "kernels.cuh"

namespace pmgpu {

RxfKernel<float> rxfwd_single3();
RxiKernel<float> rxinv_single3();
template <> RxfKernel<float> rxfwd_kernel<float, 3>(bool pairs) { return pairs ? k_rxfwd<float2, 3> : rxfwd_single3(); }
template <> RxiKernel<float> rxinv_kernel<float, 3>(bool pairs) { return pairs ? k_rxinv<float2, 3> : rxinv_single3(); }

int upload_cs_x_f32_3(const void *t32, const void *t64) { return upload_cs_local(t32, t64); }

}  // namespace pmgpu
