// passes_ct_x_f64.cu -- compile-time x passes (double fields of 3 components).
#include "kernels.cuh"

namespace pmgpu {

#define PMGPU_PLAN_X_F64(S, N, A, B, C)                                                    \
  if (lg == 12 && CtPlan<N, S, 12, A, B, C>::is(pl)) return K<double, 3, CtPlan<N, S, 12, A, B, C>>; \
  if (lg == 6 && (N * (1 + S)) > 64 && CtPlan<N, S, 6, A, B, C>::is(pl)) return K<double, 3, CtPlan<N, S, 6, A, B, C>>;

#define K k_rxfwd
template <> RxfKernel<double> rxfwd_kernel_ct<double>(const LinePlan &pl, int lg) {
#include "line_plans.inc"
  return nullptr;
}
#undef K
#define K k_rxinv
template <> RxiKernel<double> rxinv_kernel_ct<double>(const LinePlan &pl, int lg) {
#include "line_plans.inc"
  return nullptr;
}
#undef K

int upload_cs_ct_x_f64(const void *t32, const void *t64) { return upload_cs_local(t32, t64); }

}  // namespace pmgpu
