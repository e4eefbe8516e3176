// passes_ct_yi_f32.cu -- compile-time line passes (y inverse, float fields of 3 components).
#define CT_LINE float2
#define CT_MODE L_INV
#define CT_UPLOAD upload_cs_ct_yi_f32
#define PMGPU_PLAN_Y_F32 CT_PLAN
#include "lines_ct.inc"
