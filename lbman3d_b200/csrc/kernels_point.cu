// kernels_point.cu -- the shared-memory-free time step (qpoint.cuh), FP32.
#include "point_launch.cuh"

LBMAN_DEFINE_POINT_Q(f32, float)
LBMAN_DEFINE_POINT_LBM(f32, float, float, true)
