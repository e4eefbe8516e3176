// passes_lines_f32b.cu -- the register-engine batched line pass kernel for float fields.
#include "kernels.cuh"

namespace pmgpu {

template <> LinesBatchKernel<float> lines_batch_kernel<float>() { return k_lines_batch<float>; }

int upload_cs_lines_f32b(const void *t32, const void *t64) { return upload_cs_local(t32, t64); }

}  // namespace pmgpu
