// passes_x_f32_1.cu -- x passes of float fields of 1 component.
#include "kernels.cuh"

namespace pmgpu {

RxfKernel<float> rxfwd_single1();
RxiKernel<float> rxinv_single1();
template <> RxfKernel<float> rxfwd_kernel<float, 1>(bool pairs) { return pairs ? k_rxfwd<float2, 1> : rxfwd_single1(); }
template <> RxiKernel<float> rxinv_kernel<float, 1>(bool pairs) { return pairs ? k_rxinv<float2, 1> : rxinv_single1(); }

int upload_cs_x_f32_1(const void *t32, const void *t64) { return upload_cs_local(t32, t64); }

}  // namespace pmgpu
