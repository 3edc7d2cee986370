// diag_launch.cuh -- launchers of the diagnostics (reduce.cuh), instantiated by
// kernels_diag.cu (FP32 fields; the FP16-storage mode's fields are FP32) and
// kernels_diag_f64.cu.
#pragma once

#include "launch.h"
#include "reduce.cuh"

#define LBMAN_DEFINE_DIAG(SUF, R)                                                                              \
    namespace lbman {                                                                                          \
    cudaError_t launch_flow_reduce_##SUF(const SimParams& P, const void* rho, const void* u, void* upast,      \
                                         double* partials, int G, cudaStream_t st) {                           \
        flow_reduce_kernel<R><<<G, kRedThreads, 0, st>>>(P, (const R*)rho, (const R*)u, (R*)upast, partials);  \
        return cudaGetLastError();                                                                             \
    }                                                                                                          \
    cudaError_t launch_energy_reduce_##SUF(const SimParams& P, const void* q, double* partials, int G,         \
                                           cudaStream_t st) {                                                  \
        const int64_t tiles = (int64_t)((P.nx + kEnX - 1) / kEnX) * ((P.ny + kEnY - 1) / kEnY);                \
        energy_reduce_kernel<R><<<G, kRedThreads, 0, st>>>(P, diag_planes(tiles, P.zhi - P.zlo), (const R*)q,  \
                                                           partials);                                          \
        return cudaGetLastError();                                                                             \
    }                                                                                                          \
    cudaError_t launch_defects_##SUF(const SimParams& P, const void* q, uint8_t* flags,                        \
                                     unsigned long long* count, cudaStream_t st) {                             \
        if (cudaError_t e = cudaMemsetAsync(count, 0, sizeof(*count), st)) return e;                           \
        const int gx = (P.nx + kDefX - 1) / kDefX, gy = (P.ny + kDefY - 1) / kDefY;                            \
        const int zc = diag_planes((int64_t)gx * gy, P.nz);                                                    \
        const int64_t blocks = (int64_t)gx * gy * ((P.nz + zc - 1) / zc);                                      \
        defect_kernel<R><<<(unsigned)blocks, kDefThreads, 0, st>>>(P, zc, (const R*)q, flags, count);          \
        return cudaGetLastError();                                                                             \
    }                                                                                                          \
    }
