// kernels_ens_point_f64.cu -- the same for FP64 (built with --fmad=false).
#include "ens_point_impl.cuh"

LBMAN_ENS_DEFINE_QPOINT(f64, double)
LBMAN_ENS_DEFINE_LBM(f64, double, double, false)
