// kernels_ens_point.cu -- the ensemble's split organisation, FP32 and FP16 storage.
#include "ens_point_impl.cuh"

LBMAN_ENS_DEFINE_QPOINT(f32, float)
LBMAN_ENS_DEFINE_LBM(f32, float, float, true)
LBMAN_ENS_DEFINE_LBM(f16, float, __half, true)
