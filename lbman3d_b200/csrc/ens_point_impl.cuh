// ens_point_impl.cuh -- launchers of the ensemble's split organisation.
#pragma once

#include "ens_launch.h"

#define LBMAN_ENS_DEFINE_QPOINT(SUF, R)                                                                          \
    namespace lbman {                                                                                            \
    cudaError_t ens_qpoint_##SUF(const EnsBox* boxes, const EnsPointWork* work, int nwork, bool upwind, int par, \
                                 cudaStream_t st) {                                                              \
        if (upwind) ens_qpoint_kernel<R, true><<<nwork, kPointThreads, 0, st>>>(boxes, work, par);               \
        else ens_qpoint_kernel<R, false><<<nwork, kPointThreads, 0, st>>>(boxes, work, par);                     \
        return cudaGetLastError();                                                                               \
    }                                                                                                            \
    }
#define LBMAN_ENS_DEFINE_LBM(SUF, R, S, DEV)                                                                     \
    namespace lbman {                                                                                            \
    cudaError_t ens_lbm_point_##SUF(const EnsBox* boxes, const EnsLbmWork* work, int nwork, int par, int fcur,   \
                                    bool odd, bool last, cudaStream_t st) {                                      \
        auto k = odd ? ens_lbm_point_kernel<R, S, DEV, true> : ens_lbm_point_kernel<R, S, DEV, false>;           \
        k<<<nwork, kPointThreads, 0, st>>>(boxes, work, par, fcur, last ? 1 : 0);                                \
        return cudaGetLastError();                                                                               \
    }                                                                                                            \
    }
