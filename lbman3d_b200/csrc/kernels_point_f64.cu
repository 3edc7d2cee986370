// kernels_point_f64.cu -- the shared-memory-free time step (qpoint.cuh), FP64 (compiled with
// --fmad=false, as kernels_f64.cu).
#include "point_launch.cuh"

LBMAN_DEFINE_POINT_Q(f64, double)
LBMAN_DEFINE_POINT_LBM(f64, double, double, false)
