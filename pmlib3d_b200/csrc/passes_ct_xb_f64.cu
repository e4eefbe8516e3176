// passes_ct_xb_f64.cu -- batched compile-time x passes (double fields of 3 components).
#include "kernels.cuh"

namespace pmgpu {

// a batch's x tiles hold 12 or 6 vectors a point (x_shape)
static __global__ void __launch_bounds__(LINE_THREADS_MAX, LINE_CTAS) k_xf_batch_ct(BatchWork bw, BatchIo bio) {
  typedef double R;
  typedef cplx_t<R>::type C;
  __shared__ PassDesc<R> sd;
  XSmem s;
  int cur = -1, i0, i1, staged = -1;
  while (batch_next(bw, i0, i1)) {
    for (int it = i0; it < i1; it++) {
      if (cur >= 0 && (it < sd.first || it >= sd.first + sd.ntiles)) {
        cp_async_wait_all();  // no copy into the old layout may still be in flight
        staged = -1;
      }
      if (batch_patch<R>(bw, it, sd, cur)) {
        s = x_setup<double, 3>(sd.g, sd.RB, false);
        __syncthreads();
      }
      const R *in = reinterpret_cast<const R *>(bio.p[sd.patch]);
      R *stage = line_smem_at<R>(s.stage);
      if (staged != it) rxf_load<R, 3>(sd.g, in, sd.RB, sd.cs, sd.vec16, stage, it - sd.first);
      cp_async_wait_all();
      __syncthreads();
      const int next = it + 1;
      const bool pre = next < i1 && next < sd.first + sd.ntiles;
      auto prefetch = [&]() {
        if (pre) rxf_load<R, 3>(sd.g, in, sd.RB, sd.cs, sd.vec16, stage, next - sd.first);
      };
      switch (sd.cls) {
#define XTILE(S, N, LG, A, B, C) \
  case plan_class(N, S, LG): \
    rxf_tile<double, 3, CtPlan<N, S, LG, A, B, C>>(sd.g, reinterpret_cast<cplx_t<R>::type *>(sd.out), sd.RB, sd.dLG, s, \
                                               it - sd.first, prefetch); \
    break;
#define PMGPU_PLAN_X_F64(S, N, A, B, C) XTILE(S, N, 12, A, B, C) XTILE(S, N, 6, A, B, C)
#include "line_plans.inc"
#undef XTILE
        default: break;  // the part holds compile-time plans only
      }
      staged = pre ? next : -1;
    }
  }
  cp_async_wait_all();
}
static __global__ void __launch_bounds__(LINE_THREADS_MAX, LINE_CTAS) k_xi_batch_ct(BatchWork bw, BatchIo bio) {
  typedef double R;
  typedef cplx_t<R>::type C;
  __shared__ PassDesc<R> sd;
  XSmem s;
  int cur = -1, i0, i1;
  while (batch_next(bw, i0, i1)) {
    for (int it = i0; it < i1; it++) {
      if (batch_patch<R>(bw, it, sd, cur)) {
        s = x_setup<double, 3>(sd.g, sd.RB, true);
        __syncthreads();
      }
      switch (sd.cls) {
#define XTILE(S, N, LG, A, B, C) \
  case plan_class(N, S, LG): \
    rxi_tile<double, 3, CtPlan<N, S, LG, A, B, C>>(sd.g, reinterpret_cast<const cplx_t<R>::type *>(sd.in), \
                                               (R *)bio.p[sd.patch], sd.RB, sd.cs, sd.dLG, s, it - sd.first); \
    break;
#include "line_plans.inc"
#undef XTILE
        default: break;
      }
    }
  }
}
template <> RxBatchKernel rx_batch_ct<double>(bool inverse) { return inverse ? k_xi_batch_ct : k_xf_batch_ct; }

int upload_cs_ct_xb_f64(const void *t32, const void *t64) { return upload_cs_local(t32, t64); }

}  // namespace pmgpu
