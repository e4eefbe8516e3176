// passes_ct_x_f32.cu -- compile-time x passes (float fields of 3 components).
#include "kernels.cuh"

namespace pmgpu {

#define PMGPU_PLAN_X_F32(S, N, A, B, C)                                                    \
  if (lg == 12 && CtPlan<N, S, 12, A, B, C>::is(pl)) return K<float2, 3, CtPlan<N, S, 12, A, B, C>>; \
  if (lg == 6 && (N * (1 + S)) > 64 && CtPlan<N, S, 6, A, B, C>::is(pl)) return K<float2, 3, CtPlan<N, S, 6, A, B, C>>;

#define K k_rxfwd
template <> RxfKernel<float> rxfwd_kernel_ct<float>(const LinePlan &pl, int lg) {
#include "line_plans.inc"
  return nullptr;
}
#undef K
#define K k_rxinv
template <> RxiKernel<float> rxinv_kernel_ct<float>(const LinePlan &pl, int lg) {
#include "line_plans.inc"
  return nullptr;
}
#undef K

int upload_cs_ct_x_f32(const void *t32, const void *t64) { return upload_cs_local(t32, t64); }

}  // namespace pmgpu
