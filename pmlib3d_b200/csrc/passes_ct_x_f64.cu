// passes_ct_x_f64.cu -- compile-time x passes (double fields of 3 components), and the choice among
// the compile-time line passes.
#include "kernels.cuh"

namespace pmgpu {

LinesKernel<double> ct_yf_f64_kernel(const LinePlan &pl, int lg);
LinesKernel<double> ct_yi_f64_kernel(const LinePlan &pl, int lg);
LinesKernel<double> ct_z_f64_kernel(const LinePlan &pl, int lg);
template <> LinesKernel<double> lines_kernel_ct<double>(int lmode, const LinePlan &pl, int lg) {
  return lmode == L_FWD ? ct_yf_f64_kernel(pl, lg) : lmode == L_INV ? ct_yi_f64_kernel(pl, lg) : ct_z_f64_kernel(pl, lg);
}

LinesBatchCt ct_yf_f64_batch();
LinesBatchCt ct_yi_f64_batch();
LinesBatchCt ct_z_f64_batch();
template <> LinesBatchCt lines_batch_ct<double>(int lmode) {
  return lmode == L_FWD ? ct_yf_f64_batch() : lmode == L_INV ? ct_yi_f64_batch() : ct_z_f64_batch();
}

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
