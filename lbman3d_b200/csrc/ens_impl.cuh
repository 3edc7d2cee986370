// ens_impl.cuh -- launchers of the ensemble's fused kernels (ens.cuh), instantiated
// by kernels_ens.cu (FP32, FP16 storage) and kernels_ens_f64.cu (FP64, built
// with --fmad=false like the single-box FP64 path, so batched and single-box
// FP64 runs agree bit for bit).  Grids are persistent: as many blocks as fit
// on the device at once, striding through the work lists.
#pragma once
#include "ens.cuh"
#include "ens_launch.h"
#include "kernels_impl.cuh"

namespace lbman {
namespace {

template <class R, class S, bool DEV>
struct EnsImpl {
    // Resident blocks per SM of the persistent grid: the larger of the
    // occupancy query and the count from the SM's resources (the query has
    // answered low for kernels that run two blocks per SM here).
    template <class TL>
    static int occupancy() {
        int n = 0;
        const size_t smem = TL::template smem_bytes<R>();
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, ens_fused_kernel<TL, R, S, DEV, false>, TL::NT, smem) !=
            cudaSuccess)
            cudaGetLastError();
        return std::max(n, impl::fit_blocks<ens_fused_kernel<TL, R, S, DEV, false>>(TL::NT, smem));
    }

    static cudaError_t fused(const EnsFusedLaunch& L, cudaStream_t st) {
        return impl::with_tile<R>(L.tcx, L.tcy, [&](auto tl) {
            using TL = decltype(tl);
            const size_t smem = TL::template smem_bytes<R>();
            auto go = [&](auto kern) {
                kern<<<L.grid, TL::NT, smem, st>>>(L.boxes, L.work, L.nwork, L.par, L.fcur, L.first, L.write_rho_all);
            };
            if (L.upwind) go(ens_fused_kernel<TL, R, S, DEV, true>);
            else go(ens_fused_kernel<TL, R, S, DEV, false>);
            return cudaGetLastError();
        });
    }

    static cudaError_t prepare(size_t max_smem) {
        cudaError_t e = cudaSuccess;
        for (const auto& xy : kTileList) {
            const int x = xy[0], y = xy[1];
            impl::with_tile<R>(x, y, [&](auto tl) {
                using TL = decltype(tl);
                const size_t need = std::min(max_smem, TL::template smem_bytes<R>());
                auto attr = [&](auto kern) {
                    if (e == cudaSuccess)
                        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need);
                };
                attr(ens_fused_kernel<TL, R, S, DEV, true>);
                attr(ens_fused_kernel<TL, R, S, DEV, false>);
                return cudaSuccess;
            });
        }
        return e;
    }

    static int blocks_per_sm(int tcx, int tcy) {
        int n = 0;
        impl::with_tile<R>(tcx, tcy, [&](auto tl) {
            n = occupancy<decltype(tl)>();
            return cudaSuccess;
        });
        return n;
    }
};

}  // namespace

}  // namespace lbman

#define LBMAN_ENS_DEFINE(SUF, R, S, DEV)                                                                 \
    namespace lbman {                                                                                     \
    LBMAN_ENS_DEFINE_BODY(SUF, R, S, DEV)                                                                 \
    }

namespace lbman {
#define LBMAN_ENS_DEFINE_BODY(SUF, R, S, DEV)                                                                       \
    cudaError_t ens_fused_##SUF(const EnsFusedLaunch& L, cudaStream_t st) { return EnsImpl<R, S, DEV>::fused(L, st); } \
    cudaError_t ens_prepare_##SUF(size_t s) { return EnsImpl<R, S, DEV>::prepare(s); }                              \
    int ens_blocks_per_sm_##SUF(int x, int y) { return EnsImpl<R, S, DEV>::blocks_per_sm(x, y); }

}  // namespace lbman
