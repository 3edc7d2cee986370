// kernels_diag.cu -- diagnostics of FP32 fields.
#include "diag_launch.cuh"

LBMAN_DEFINE_DIAG(f32, float)
