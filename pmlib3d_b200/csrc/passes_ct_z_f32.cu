// passes_ct_z_f32.cu -- compile-time line passes (z, float fields of 3 components).
#define CT_LINE float2
#define CT_MODE L_Z
#define CT_UPLOAD upload_cs_ct_z_f32
#define PMGPU_PLAN_Z_F32 CT_PLAN
#include "lines_ct.inc"
