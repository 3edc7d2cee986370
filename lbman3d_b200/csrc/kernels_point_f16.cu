// kernels_point_f16.cu -- the shared-memory-free time step (qpoint.cuh), FP16 storage
// (its Q stage is the FP32 one).
#include "point_launch.cuh"

LBMAN_DEFINE_POINT_LBM(f16, float, __half, true)
