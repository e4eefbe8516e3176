// passes_x_f32_s.cu -- x passes of float fields whose rows are too long for two rows a vector.
#include "kernels.cuh"

namespace pmgpu {

RxfKernel<float> rxfwd_single1() { return k_rxfwd<float, 1>; }
RxiKernel<float> rxinv_single1() { return k_rxinv<float, 1>; }
RxfKernel<float> rxfwd_single3() { return k_rxfwd<float, 3>; }
RxiKernel<float> rxinv_single3() { return k_rxinv<float, 3>; }

int upload_cs_x_f32_s(const void *t32, const void *t64) { return upload_cs_local(t32, t64); }

}  // namespace pmgpu
