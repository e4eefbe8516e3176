// passes_ct_xb_f32.cu -- batched compile-time x passes (float fields of 3 components).
#define CT_LINE float2
#define CT_UPLOAD upload_cs_ct_xb_f32
#define PMGPU_PLAN_X_F32 CT_PLAN
#include "x_batch_ct.inc"
