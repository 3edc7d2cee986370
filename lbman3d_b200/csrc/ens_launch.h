// ens_launch.h -- host-side launchers of the ensemble kernels (kernels_ens*.cu:
// the fused organisation; kernels_ens_point*.cu: the split one).
#pragma once

#include <cuda_runtime.h>

#include "ens.cuh"

namespace lbman {

// One fused launch over every box of an ensemble.
struct EnsFusedLaunch {
    const EnsBox* boxes;
    const EnsQWork* work;
    int nwork;
    int tcx, tcy;
    bool upwind;
    int par, fcur, first, write_rho_all;
    int grid;
};

#define LBMAN_ENS_DECLARE(SUF)                                                                                \
    cudaError_t ens_fused_##SUF(const EnsFusedLaunch& L, cudaStream_t st);                                    \
    cudaError_t ens_prepare_##SUF(size_t max_smem);                                                           \
    int ens_blocks_per_sm_##SUF(int tcx, int tcy);                                                            \
    cudaError_t ens_qpoint_##SUF(const EnsBox* boxes, const EnsPointWork* work, int nwork, bool upwind, int par, \
                                 cudaStream_t st);                                                            \
    cudaError_t ens_lbm_point_##SUF(const EnsBox* boxes, const EnsLbmWork* work, int nwork, int par, int fcur, \
                                    bool odd, bool last, cudaStream_t st);

LBMAN_ENS_DECLARE(f64)
LBMAN_ENS_DECLARE(f32)
LBMAN_ENS_DECLARE(f16)

}  // namespace lbman
