// passes_ct_z_f64.cu -- compile-time line passes (z, double fields of 3 components).
#define CT_LINE double
#define CT_MODE L_Z
#define CT_UPLOAD upload_cs_ct_z_f64
#define PMGPU_PLAN_Z_F64 CT_PLAN
#include "lines_ct.inc"
