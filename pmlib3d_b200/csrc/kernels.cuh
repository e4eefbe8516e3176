// kernels.cuh -- the pass kernels as the launchers (passes.cuh) reach them.  Every kernel is
// compiled in one of the passes_*.cu units, so that they build in parallel and a change
// of the launchers does not rebuild them.
#pragma once

#include "host.h"
#include "solve.cuh"

namespace pmgpu {

// a line-pass kernel (k_rlines); pairs: FP32 tiles of two lines a vector.  Defined in
// the lines_*.cu units.
template <typename R>
using LinesKernel = void (*)(SolveGeom<R>, LineTiles, const typename cplx_t<R>::type *, typename cplx_t<R>::type *,
                             int, int, int, int, int, int);
template <typename R> LinesKernel<R> lines_kernel(bool pairs);
template <> LinesKernel<float> lines_kernel<float>(bool pairs);
template <> LinesKernel<double> lines_kernel<double>(bool pairs);
// the batched line-pass kernel (k_lines_batch)
template <typename R> using LinesBatchKernel = void (*)(BatchWork, int, int, int);
template <typename R> LinesBatchKernel<R> lines_batch_kernel();
template <> LinesBatchKernel<float> lines_batch_kernel<float>();
template <> LinesBatchKernel<double> lines_batch_kernel<double>();

// ---- compile-time line passes (k_rlines_ct), one unit a mode and type: lines_ct.inc
typedef void (*LinesBatchCt)(BatchWork);
// Vectors a position of a plan's tiles, as line_shape picks them without a tuned tile;
// slack: 0, or BATCH_SMEM_SLACK in a batch
template <int LMODE, int S, int N, int A, int B, int C> constexpr int ct_vectors(size_t slack) {
  typedef CtPlan<N, S, 12, A, B, C> PL;
  return line_whole_block(line_tab_bytes(N, PL::twiddles(), S != 0, A, 16) + 12 * 16 * (size_t)N * (1 + S) + slack,
                          LMODE == L_Z && slack == 0)
             ? 12
             : 6;
}
template <int LMODE, int S, int N, int A, int B, int C>
using CtSingle = CtPlan<N, S, ct_vectors<LMODE, S, N, A, B, C>(0), A, B, C>;
template <int LMODE, int S, int N, int A, int B, int C>
using CtBatch = CtPlan<N, S, ct_vectors<LMODE, S, N, A, B, C>(BATCH_SMEM_SLACK), A, B, C>;
// the kernel of plan pl with lg vectors a position, nullptr if there is none
template <typename T, int LMODE> LinesKernel<typename LineT<T>::R> ct_lines(const LinePlan &pl, int lg);
// the batched kernel, and the class of a plan in it: 0 if its switch does not hold the plan
template <typename T, int LMODE> LinesBatchCt ct_lines_batch();
template <typename T, int LMODE> int ct_lines_class(const LinePlan &pl, int lg);
#define PMGPU_CT_LINES(T, M)                                                             \
  template <> LinesKernel<LineT<T>::R> ct_lines<T, M>(const LinePlan &, int);            \
  template <> LinesBatchCt ct_lines_batch<T, M>();                                       \
  template <> int ct_lines_class<T, M>(const LinePlan &, int);
PMGPU_CT_LINES(float2, L_FWD) PMGPU_CT_LINES(float2, L_INV) PMGPU_CT_LINES(float2, L_Z)
PMGPU_CT_LINES(double, L_FWD) PMGPU_CT_LINES(double, L_INV) PMGPU_CT_LINES(double, L_Z)
#undef PMGPU_CT_LINES
template <typename R> inline LinesKernel<R> lines_kernel_ct(int lmode, const LinePlan &pl, int lg) {
  typedef typename StockLine<R>::T T;
  return lmode == L_FWD ? ct_lines<T, L_FWD>(pl, lg) : lmode == L_INV ? ct_lines<T, L_INV>(pl, lg) : ct_lines<T, L_Z>(pl, lg);
}
template <typename R> inline LinesBatchCt lines_batch_ct(int lmode) {
  typedef typename StockLine<R>::T T;
  return lmode == L_FWD ? ct_lines_batch<T, L_FWD>() : lmode == L_INV ? ct_lines_batch<T, L_INV>() : ct_lines_batch<T, L_Z>();
}
template <typename R> inline int lines_batch_class(int lmode, const LinePlan &pl, int lg) {
  typedef typename StockLine<R>::T T;
  return lmode == L_FWD ? ct_lines_class<T, L_FWD>(pl, lg)
                        : lmode == L_INV ? ct_lines_class<T, L_INV>(pl, lg) : ct_lines_class<T, L_Z>(pl, lg);
}

// x-pass kernels (k_rxfwd, k_rxinv and their batched forms); pairs: FP32 vectors of two
// rows.  Defined in the passes_x*.cu units.
template <typename R>
using RxfKernel = void (*)(SolveGeom<R>, const R *, typename cplx_t<R>::type *, int, int, int, FastDiv);
template <typename R>
using RxiKernel = void (*)(SolveGeom<R>, const typename cplx_t<R>::type *, R *, int, int, FastDiv);
using RxBatchKernel = void (*)(BatchWork, BatchIo);
template <typename R, int NC> RxfKernel<R> rxfwd_kernel(bool pairs);
template <typename R, int NC> RxiKernel<R> rxinv_kernel(bool pairs);
template <> RxfKernel<float> rxfwd_kernel<float, 1>(bool);
template <> RxfKernel<float> rxfwd_kernel<float, 3>(bool);
template <> RxfKernel<double> rxfwd_kernel<double, 1>(bool);
template <> RxfKernel<double> rxfwd_kernel<double, 3>(bool);
template <> RxiKernel<float> rxinv_kernel<float, 1>(bool);
template <> RxiKernel<float> rxinv_kernel<float, 3>(bool);
template <> RxiKernel<double> rxinv_kernel<double, 1>(bool);
template <> RxiKernel<double> rxinv_kernel<double, 3>(bool);
// compile-time kernels of 3-component x passes with lg vectors a point (nullptr: none)
template <typename R> RxfKernel<R> rxfwd_kernel_ct(const LinePlan &pl, int lg);
template <typename R> RxiKernel<R> rxinv_kernel_ct(const LinePlan &pl, int lg);
template <> RxfKernel<float> rxfwd_kernel_ct<float>(const LinePlan &, int);
template <> RxfKernel<double> rxfwd_kernel_ct<double>(const LinePlan &, int);
template <> RxiKernel<float> rxinv_kernel_ct<float>(const LinePlan &, int);
template <> RxiKernel<double> rxinv_kernel_ct<double>(const LinePlan &, int);
template <typename R> RxBatchKernel rx_batch_kernel(bool inverse);
// the batched compile-time kernel, and the class of a plan in it (0: none)
template <typename R> RxBatchKernel rx_batch_ct(bool inverse);
template <typename R> int rx_batch_class(const LinePlan &pl, int lg);
template <> int rx_batch_class<float>(const LinePlan &, int);
template <> int rx_batch_class<double>(const LinePlan &, int);
template <> RxBatchKernel rx_batch_ct<float>(bool);
template <> RxBatchKernel rx_batch_ct<double>(bool);
template <> RxBatchKernel rx_batch_kernel<float>(bool);
template <> RxBatchKernel rx_batch_kernel<double>(bool);

// copies the DFT constant tables into this unit's constant memory
static int upload_cs_local(const void *t32, const void *t64) {
  if (cudaMemcpyToSymbol(c_cs32, t32, sizeof(c_cs32)) != cudaSuccess) return -1;
  if (cudaMemcpyToSymbol(c_cs64, t64, sizeof(c_cs64)) != cudaSuccess) return -1;
  return 0;
}

}  // namespace pmgpu
