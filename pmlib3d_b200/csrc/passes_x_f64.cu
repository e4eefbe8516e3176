// passes_x_f64.cu -- x passes of double fields.
#include "kernels.cuh"

namespace pmgpu {

template <> RxfKernel<double> rxfwd_kernel<double, 1>(bool) { return k_rxfwd<double, 1>; }
template <> RxfKernel<double> rxfwd_kernel<double, 3>(bool) { return k_rxfwd<double, 3>; }
template <> RxiKernel<double> rxinv_kernel<double, 1>(bool) { return k_rxinv<double, 1>; }
template <> RxiKernel<double> rxinv_kernel<double, 3>(bool) { return k_rxinv<double, 3>; }

int upload_cs_x_f64(const void *t32, const void *t64) { return upload_cs_local(t32, t64); }

}  // namespace pmgpu
