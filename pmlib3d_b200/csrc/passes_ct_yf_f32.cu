// passes_ct_yf_f32.cu -- compile-time line passes (y forward, float fields of 3 components).
#define CT_LINE float2
#define CT_MODE L_FWD
#define CT_UPLOAD upload_cs_ct_yf_f32
#define PMGPU_PLAN_Y_F32 CT_PLAN
#include "lines_ct.inc"
