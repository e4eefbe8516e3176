// passes_lines_f32.cu -- the register-engine line pass kernel for float fields.
#include "kernels.cuh"

namespace pmgpu {

template <> LinesKernel<float> lines_kernel<float>(bool pairs) { return pairs ? k_rlines<float2> : k_rlines<float>; }

int upload_cs_lines_f32(const void *t32, const void *t64) { return upload_cs_local(t32, t64); }

}  // namespace pmgpu
