// point_launch.cuh -- launchers of the qpoint.cuh kernels, instantiated by
// kernels_point.cu (FP32), kernels_point_f16.cu (FP16 storage: the LBM step
// only) and kernels_point_f64.cu.
#pragma once

#include "launch.h"
#include "pdl.cuh"
#include "qpoint.cuh"

#include <algorithm>

namespace lbman {
namespace impl {

// The compiled wall-rule masks, each a superset of the ones before: none, x
// walls (slit), x and y walls (channel), everything.
inline int point_mask(const SimParams& P) {
    int m = 0;
    for (int ax = 0; ax < 3; ++ax) {
        if (!(P.qper[2 * ax] && P.qper[2 * ax + 1] && P.uper[2 * ax] && P.uper[2 * ax + 1])) m |= 1 << ax;
        for (int f = 2 * ax; f < 2 * ax + 2; ++f)
            if (P.face[f].qbc == Q_ANCHORING) m |= QW_ANCHOR;
    }
    return m == 0 ? 0 : m == QW_X ? QW_X : (m & ~(QW_X | QW_Y)) == 0 ? QW_X | QW_Y : 15;
}
template <class F>
void with_mask(int m, F&& f) {
    if (m == 0) f(std::integral_constant<int, 0>{});
    else if (m == QW_X) f(std::integral_constant<int, QW_X>{});
    else if (m == (QW_X | QW_Y)) f(std::integral_constant<int, QW_X | QW_Y>{});
    else f(std::integral_constant<int, 15>{});
}

constexpr int kMaxGridY = 65535;

// Planes per thread (a power of two): the longest walk that still gives every
// SM a few blocks.  At most 4 planes, where the gain of reusing the centre
// values ends, and 16 blocks per SM; packed kernels on planes of 2^15 cells and
// more (long_walks), where the walk prefetches and in FP32 saves the z terms' trip
// through memory, at most 16 planes and 6 blocks per SM.  FP32 steps with walks
// of at most 4 / 8 / 16 planes there: 256x256x64 226 / 220 / 217 us, 240x160x165
// 356 / 331 / 331 us, 256^3 909 / 855 / 840 us, 512x512x128 1780 / 1680 / 1670 us.
// A box of so many planes that its chunks would pass the launch's y dimension
// walks further.
inline int point_walk(const SimParams& P, bool pair, int num_sms) {
    const bool longer = pair && long_walks(P);
    const int per_block = kPointThreads * (pair ? 2 : 1);
    const int64_t cols = (P.nxy + per_block - 1) / per_block, blocks = (int64_t)(longer ? 6 : 16) * num_sms;
    int zc = longer ? 16 : 4;
    while (zc > 1 && cols * ((P.nz + zc - 1) / zc) < blocks) zc /= 2;
    while ((P.nz + zc - 1) / zc > kMaxGridY) zc *= 2;
    return zc;
}

template <class R>
cudaError_t qpoint(const SimParams& P, bool pair, int num_sms, const void* qin, const void* uin, void* qout,
                   void* stress, void* F, cudaStream_t st) {
    const FastDiv dnx = make_fastdiv((uint32_t)P.nx);
    const int per_block = kPointThreads * (pair ? 2 : 1);
    const int zc = point_walk(P, pair, num_sms);
    const dim3 g((unsigned)((P.nxy + per_block - 1) / per_block), (unsigned)((P.nz + zc - 1) / zc));
    cudaError_t err = cudaErrorInvalidValue;
    auto launch = [&](auto k) {
        err = launch_dependent(k, g, kPointThreads, 0, st, P, dnx, zc, (const R*)qin, (const R*)uin, (R*)qout, (R*)stress,
                               (R*)F);
    };
    with_mask(point_mask(P), [&](auto m) {
        constexpr int QW = decltype(m)::value;
        if constexpr (sizeof(R) == 4) {
            if (pair) {
                auto go = [&](auto walk) {
                    constexpr int W = decltype(walk)::value;
                    if (P.upwind) launch(qpoint2_kernel<true, QW, W>);
                    else launch(qpoint2_kernel<false, QW, W>);
                };
                if (force_in_walk(P)) go(std::integral_constant<int, WALK_FORCE>{});
                else if (long_walks(P)) go(std::integral_constant<int, WALK_LONG>{});
                else go(std::integral_constant<int, WALK_SHORT>{});
                return;
            }
        }
        if (P.upwind) launch(qpoint_kernel<R, true, QW>);
        else launch(qpoint_kernel<R, false, QW>);
    });
    return err;
}

template <class R>
cudaError_t point_force(const SimParams& P, bool pair, int num_sms, const void* qn, const void* stress, const void* u,
                        void* F, cudaStream_t st) {
    const FastDiv dnx = make_fastdiv((uint32_t)P.nx), dnxy = make_fastdiv((uint32_t)P.nxy);
    const unsigned nb = (unsigned)((P.V + 255) / 256);
    const int zm = point_walk(P, pair, num_sms) - 1;
    cudaError_t err = cudaErrorInvalidValue;
    auto launch = [&](auto k) {
        err = launch_dependent(k, dim3(nb), 256, 0, st, P, dnx, dnxy, zm, (const R*)qn, (const R*)stress, (const R*)u, (R*)F);
    };
    with_mask(point_mask(P), [&](auto m) {
        constexpr int QW = decltype(m)::value;
        if constexpr (sizeof(R) == 4) {
            if (pair) {
                launch(force_in_walk(P) ? point_force_kernel<R, QW, true, true> : point_force_kernel<R, QW, true, false>);
                return;
            }
        }
        launch(point_force_kernel<R, QW, false>);
    });
    return err;
}

template <class R, class S, bool DEV>
cudaError_t lbm_aa_point(const SimParams& P, bool pair, int num_sms, bool odd, bool last, void* f, const void* qn,
                         const void* stress, void* F, void* rho, void* u, cudaStream_t st) {
    const FastDiv dnx = make_fastdiv((uint32_t)P.nx), dnxy = make_fastdiv((uint32_t)P.nxy);
    const unsigned nb = (unsigned)((P.V + kPointThreads - 1) / kPointThreads);
    const int zm = point_walk(P, pair, num_sms) - 1;
    cudaError_t err = cudaErrorInvalidValue;
    auto launch = [&](auto k) {
        err = launch_dependent(k, dim3(nb), kPointThreads, 0, st, P, dnx, dnxy, zm, (S*)f, (const R*)qn,
                               (const R*)stress, (R*)F, (R*)rho, (R*)u, last ? 1 : 0);
    };
    with_mask(point_mask(P), [&](auto m) {
        constexpr int QW = decltype(m)::value, WM = QW & 7;
        if constexpr (sizeof(R) == 4) {
            if (pair) {
                if constexpr (!std::is_same<S, __half>::value) {
                    if (force_in_walk(P)) {
                        if (odd) launch(lbm_aa_point_kernel<R, S, DEV, WM, QW, true, true, true>);
                        else launch(lbm_aa_point_kernel<R, S, DEV, WM, QW, false, true, true>);
                        return;
                    }
                } else if constexpr (QW == 0) {
                    if (long_walks(P)) {
                        // two cells per thread (the packed kernels' boxes have an even nx)
                        err = launch_dependent(odd ? lbm_aa_point_h2_kernel<DEV, true> : lbm_aa_point_h2_kernel<DEV, false>,
                                               dim3((unsigned)((P.V / 2 + 255) / 256)), 256, 0, st, P, dnx, dnxy, (S*)f,
                                               (const R*)stress, (R*)F, (R*)rho, (R*)u, last ? 1 : 0);
                        return;
                    }
                }
                if (odd) launch(lbm_aa_point_kernel<R, S, DEV, WM, QW, true, true>);
                else launch(lbm_aa_point_kernel<R, S, DEV, WM, QW, false, true>);
                return;
            }
        }
        if (odd) launch(lbm_aa_point_kernel<R, S, DEV, WM, QW, true, false>);
        else launch(lbm_aa_point_kernel<R, S, DEV, WM, QW, false, false>);
    });
    return err;
}

}  // namespace impl
}  // namespace lbman

#define LBMAN_DEFINE_POINT_Q(SUF, R)                                                                              \
    namespace lbman {                                                                                             \
    cudaError_t launch_qpoint_##SUF(const SimParams& P, bool pair, int num_sms, const void* qin, const void* uin, \
                                    void* qout, void* stress, void* F, cudaStream_t st) {                         \
        return impl::qpoint<R>(P, pair, num_sms, qin, uin, qout, stress, F, st);                                  \
    }                                                                                                             \
    cudaError_t launch_point_force_##SUF(const SimParams& P, bool pair, int num_sms, const void* qn,              \
                                         const void* stress, const void* u, void* F, cudaStream_t st) {           \
        return impl::point_force<R>(P, pair, num_sms, qn, stress, u, F, st);                                      \
    }                                                                                                             \
    }
#define LBMAN_DEFINE_POINT_LBM(SUF, R, S, DEV)                                                                    \
    namespace lbman {                                                                                             \
    cudaError_t launch_lbm_aa_point_##SUF(const SimParams& P, bool pair, int num_sms, bool odd, bool last,        \
                                          void* f, const void* qn, const void* stress, void* F, void* rho,        \
                                          void* u, cudaStream_t st) {                                             \
        return impl::lbm_aa_point<R, S, DEV>(P, pair, num_sms, odd, last, f, qn, stress, F, rho, u, st);          \
    }                                                                                                             \
    }
