// passes_ct_yi_f64.cu -- compile-time line passes (y inverse, double fields of 3 components).
#define CT_LINE double
#define CT_MODE L_INV
#define CT_UPLOAD upload_cs_ct_yi_f64
#define PMGPU_PLAN_Y_F64 CT_PLAN
#include "lines_ct.inc"
