// passes_lines_f64.cu -- the register-engine line pass kernel for double fields.
#include "kernels.cuh"

namespace pmgpu {

template <> LinesKernel<double> lines_kernel<double>(bool) { return k_rlines<double>; }

int upload_cs_lines_f64(const void *t32, const void *t64) { return upload_cs_local(t32, t64); }

}  // namespace pmgpu
