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
// the compile-time kernel of plan pl with lg vectors a position (k_rlines_ct), nullptr if
// there is none; passes_ct_*.cu
template <typename R> LinesKernel<R> lines_kernel_ct(int lmode, const LinePlan &pl, int lg);
template <> LinesKernel<float> lines_kernel_ct<float>(int, const LinePlan &, int);
template <> LinesKernel<double> lines_kernel_ct<double>(int, const LinePlan &, int);
// the batched line-pass kernel (k_lines_batch)
template <typename R> using LinesBatchKernel = void (*)(BatchWork, int, int, int);
template <typename R> LinesBatchKernel<R> lines_batch_kernel();
// batched kernels over the compile-time plans, and whether a plan is one of them
typedef void (*LinesBatchCt)(BatchWork);
template <typename R> LinesBatchCt lines_batch_ct(int lmode);
template <> LinesBatchCt lines_batch_ct<float>(int);
template <> LinesBatchCt lines_batch_ct<double>(int);
template <> LinesBatchKernel<float> lines_batch_kernel<float>();
template <> LinesBatchKernel<double> lines_batch_kernel<double>();
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
template <typename R> RxBatchKernel rx_batch_ct(bool inverse);
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
