// passes_ct_z_f64.cu -- compile-time line passes (z, double fields of 3 components).
#include "kernels.cuh"

namespace pmgpu {

// vectors a position as line_shape picks them
__host__ __device__ static constexpr int ct_lg(int points) { return points * 192 <= 104 * 1024 ? 12 : 6; }
__host__ __device__ static constexpr int bt_lg(int points) { return points * 192 <= 49 * 1024 ? 12 : 6; }  // in batches

#define PMGPU_PLAN_Z_F64(S, N, A, B, C)                                                  \
  if (lg == ct_lg(N * (1 + S)) && CtPlan<N, S, ct_lg(N * (1 + S)), A, B, C>::is(pl))      \
    return k_rlines_ct<double, L_Z, CtPlan<N, S, ct_lg(N * (1 + S)), A, B, C>>;               \
  if (lg == bt_lg(N * (1 + S)) && CtPlan<N, S, bt_lg(N * (1 + S)), A, B, C>::is(pl))      \
    return k_rlines_ct<double, L_Z, CtPlan<N, S, bt_lg(N * (1 + S)), A, B, C>>;

LinesKernel<double> ct_z_f64_kernel(const LinePlan &pl, int lg) {
#include "line_plans.inc"
  return nullptr;
}

#undef PMGPU_PLAN_Z_F64

// the same plans in a batch: a patch's class picks the tile function
static __global__ void __launch_bounds__(LINE_THREADS_MAX, LINE_CTAS) k_z_batch_ct(BatchWork bw) {
  typedef cplx_t<double>::type C;
  __shared__ PassDesc<double> sd;
  LineSmem s;
  int cur = -1, i0, i1;
  while (batch_next(bw, i0, i1)) {
    for (int it = i0; it < i1; it++) {
      if (batch_patch<double>(bw, it, sd, cur)) {
        s = line_setup<double>(sd.g, 2, L_Z);
        __syncthreads();
      }
      int o, k0;
      line_tile_at(sd.lt, it - sd.first, sd.lt.TK, o, k0);
      const LineIo<double> io = line_io<double>(sd.lt, reinterpret_cast<const C *>(sd.in), reinterpret_cast<C *>(sd.out), 3, o, k0);
      switch (sd.cls) {
#define PMGPU_PLAN_Z_F64(S, N, A, B, C)             \
  case plan_class(N, S, bt_lg(N * (1 + S))):           \
    line_tile_ct<double, L_Z, CtPlan<N, S, bt_lg(N * (1 + S)), A, B, C>>(sd.g, io, s.tabs, o, k0); break;
#include "line_plans.inc"
        default: break;  // the part holds compile-time plans only
      }
    }
  }
}
LinesBatchCt ct_z_f64_batch() { return k_z_batch_ct; }

int upload_cs_ct_z_f64(const void *t32, const void *t64) { return upload_cs_local(t32, t64); }

}  // namespace pmgpu
