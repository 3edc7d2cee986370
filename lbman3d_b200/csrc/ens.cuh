// ens.cuh -- ensemble kernels: many independent boxes of different sizes,
// boundary configurations and physical parameters advanced together.
//
// Every box is described by an EnsBox in device memory (its own SimParams
// and field pointers).  The host flattens all boxes into work lists, and each
// launch covers every box, running the code of the single-box kernels on the
// item's box: one point per thread, so the results are bit for bit those of a
// single box with the one-point kernels (FP64, LBMAN_KERNELS_SPLIT, and AUTO
// where its 30-wide tiles do not fit; the packed arithmetic of the other FP32 and
// FP16 boxes rounds differently).  There is no communication between boxes.
//
//   split   ens_qpoint_kernel, then ens_lbm_point_kernel (the time step of
//           qpoint.cuh, in-place streaming): one block per work item;
//   fused   ens_fused_kernel (fused.cuh): a persistent grid of z-marching blocks
//           strides through the list.
//
// A time step of the whole ensemble is therefore two launches (split) or one
// (fused), which the host replays from a CUDA graph.
#pragma once

#include "fused.cuh"
#include "lbm.cuh"
#include "qpoint.cuh"

namespace lbman {

struct EnsBox {
    SimParams P;
    FastDiv dnx, dnxy;
    void* q[2];   // Q, double buffered
    void* u[2];   // u, double buffered (fused); the split organisation uses u[0] only
    void* f[2];   // populations; the second buffer only for the fused organisation
    void* rho;
    void* F;
    void* stress; // between the split organisation's two kernels
    int zc;       // z chunk of this box's fused work items
    int mask;     // wall-rule mask of the split kernels (point_mask)
};
static_assert(sizeof(EnsBox) % 4 == 0, "copied to shared memory as 32-bit words");

struct EnsQWork {
    int box, bx, by, bz;
};
struct EnsPointWork {
    int box, block, z0, z1;  // 128 columns of the planes [z0, z1)
};
struct EnsLbmWork {
    int box, block;  // kEnsLbmCells cells
};

// A work item's box, copied to shared memory: a single-box launch reads its
// parameters from the constant bank, a global-memory copy would cost a load
// per use.
__device__ __forceinline__ const EnsBox& ens_box(const EnsBox* __restrict__ boxes, int box, uint32_t* buf) {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(boxes + box);
    for (int i = threadIdx.x; i < (int)(sizeof(EnsBox) / 4); i += blockDim.x) buf[i] = src[i];
    __syncthreads();
    return *reinterpret_cast<const EnsBox*>(buf);
}

// Calls f with the compile-time mask that `mask` (block-uniform) names.
template <class F>
__device__ __forceinline__ void ens_with_mask(int mask, F&& f) {
    if (mask == 0) f(std::integral_constant<int, 0>{});
    else if (mask == QW_X) f(std::integral_constant<int, QW_X>{});
    else if (mask == (QW_X | QW_Y)) f(std::integral_constant<int, QW_X | QW_Y>{});
    else f(std::integral_constant<int, 15>{});
}

template <class R, bool UPWIND>
__global__ void __launch_bounds__(kPointThreads, point_min_blocks<R>())
    ens_qpoint_kernel(const EnsBox* __restrict__ boxes, const EnsPointWork* __restrict__ work, int par) {
    __shared__ __align__(16) uint32_t buf[sizeof(EnsBox) / 4];
    const EnsPointWork it = work[blockIdx.x];
    const EnsBox& B = ens_box(boxes, it.box, buf);
    const SimParams& P = B.P;
    const int n = (int)P.nxy;
    int col = it.block * kPointThreads + threadIdx.x;
    const bool live = col < n;
    if (!live) col = n - 1;
    const int y = (int)fdiv((uint32_t)col, B.dnx), x = col - y * P.nx;
    ens_with_mask(B.mask, [&](auto m) {
        qpoint_column<R, UPWIND, decltype(m)::value>(P, x, y, col, it.z0, it.z1, live, (const R*)B.q[par],
                                                     (const R*)B.u[0], (R*)B.q[1 - par], (R*)B.stress, (R*)B.F);
    });
}

// Cells of an LBM work item: enough that the box's parameters are copied once
// per 4 cells of a thread.
constexpr int kEnsLbmCells = 4 * kPointThreads;

// par: the buffer holding Q_new.  HBM bound; its registers are held to 8 blocks
// per SM in FP32 and 4 in FP64.  Steps of 96 boxes (18.1 M cells) unbounded (3
// blocks) / 4 / 8: FP32 1200 / 1160 / 1145 us, FP16 storage 1065 / 1080 / 1045 us;
// FP64 2500 / 2410 us at 4.
template <class R, class S, bool DEV, bool ODD>
__global__ void __launch_bounds__(kPointThreads, sizeof(R) == 4 ? 8 : 4)
    ens_lbm_point_kernel(const EnsBox* __restrict__ boxes, const EnsLbmWork* __restrict__ work, int par, int fcur,
                         int last) {
    __shared__ __align__(16) uint32_t buf[sizeof(EnsBox) / 4];
    const EnsLbmWork it = work[blockIdx.x];
    const EnsBox& B = ens_box(boxes, it.box, buf);
    const SimParams& P = B.P;
    const int c0 = it.block * kEnsLbmCells + threadIdx.x, c1 = min((it.block + 1) * kEnsLbmCells, (int)P.V);
    S* f = (S*)(fcur ? B.f[1] : B.f[0]);
    const R* qn = (const R*)(par ? B.q[1] : B.q[0]);
    ens_with_mask(B.mask, [&](auto m) {
        constexpr int QW = decltype(m)::value, WM = QW & 7;
        const KeptPointForce<R, QW, false> force{
            {P, 0, qn, (const R*)B.stress, (const R*)B.u[0], (const R*)B.F}, (R*)B.F, last};
#pragma unroll 1
        for (int c = c0; c < c1; c += kPointThreads) {
            if constexpr (ODD)
                aa_odd_cell<R, S, DEV, WM, int>(P, B.dnx, B.dnxy, c, f, force, (R*)B.rho, (R*)B.u[0], last);
            else
                aa_even_cell<R, S, DEV, WM, int>(P, B.dnx, B.dnxy, c, f, force, (R*)B.rho, (R*)B.u[0], last);
        }
    });
}

template <class TL, class R, class S, bool DEV, bool UPWIND>
__global__ void __launch_bounds__(TL::NT) ens_fused_kernel(const EnsBox* __restrict__ boxes,
                                                           const EnsQWork* __restrict__ work, int nwork, int par,
                                                           int fcur, int first, int write_rho_all) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const EnsQWork it = work[w];
        const EnsBox& B = boxes[it.box];
        const int z0 = it.bz * B.zc;
        if (z0 < B.P.nz)
            qf_march<TL, R, UPWIND>(B.P, it.bx * TL::TCX, it.by * TL::TCY, z0, min(z0 + B.zc, B.P.nz),
                                    (const R*)B.q[par], (const R*)B.u[par], reinterpret_cast<R*>(smem_raw),
                                    CollideCell<R, S, DEV>{B.P, phys_ref<R>(B.P), first, (R*)B.q[1 - par],
                                                           (R*)B.u[1 - par], (const S*)B.f[fcur],
                                                           (S*)B.f[1 - fcur], (R*)B.rho, nullptr, write_rho_all});
        __syncthreads();
    }
}

}  // namespace lbman
