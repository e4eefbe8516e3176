// passes_lines_f64b.cu -- the register-engine batched line pass kernel for double fields.
#include "kernels.cuh"

namespace pmgpu {

template <> LinesBatchKernel<double> lines_batch_kernel<double>() { return k_lines_batch<double>; }

int upload_cs_lines_f64b(const void *t32, const void *t64) { return upload_cs_local(t32, t64); }

}  // namespace pmgpu
