// passes_ct_xb_f64.cu -- batched compile-time x passes (double fields of 3 components).
#define CT_LINE double
#define CT_UPLOAD upload_cs_ct_xb_f64
#define PMGPU_PLAN_X_F64 CT_PLAN
#include "x_batch_ct.inc"
