// stats.cu -- flow and order statistics of one box: kinetic-energy spectrum,
// Q-tensor autocorrelation and correlation length, mean / rms speed.  No
// counterpart in the reference (its analysis stops at the defect finder,
// src/analysis/defect_finder.tpp); definitions are stated in stats.h and in
// the C header.
//
// Transforms are cuFFT 3D real-to-complex (library FFTs, like cuBLAS for a
// plain GEMM); the power accumulation and the shell binning are kernels of
// this file.  Shell sums are accumulated in FP64: per block in shared memory,
// then folded over blocks in a fixed order.
#include <cufft.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "stats.h"

namespace lbman {
namespace stats {

namespace {

constexpr int kThreads = 256;

// P = |A|^2 (mode 0), P += |A|^2 (1), P = 2|A|^2 + 2|B|^2 + 2 Re(A conj B) (2),
// P += 2|A|^2 (3), A = P + 2|A|^2 as a complex number (4).
template <class R, class C>
__global__ void __launch_bounds__(kThreads) power_kernel(C* __restrict__ A, const C* __restrict__ B,
                                                         R* __restrict__ P, int64_t n, int mode) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const C a = A[i];
        const R pa = a.x * a.x + a.y * a.y;
        if (mode == 0) {
            P[i] = pa;
        } else if (mode == 1) {
            P[i] += pa;
        } else if (mode == 2) {
            const C b = B[i];
            P[i] = R(2) * pa + R(2) * (b.x * b.x + b.y * b.y) + R(2) * (a.x * b.x + a.y * b.y);
        } else if (mode == 3) {
            P[i] += R(2) * pa;
        } else {
            C c;
            c.x = P[i] + R(2) * pa;
            c.y = R(0);
            A[i] = c;
        }
    }
}

// Sum of v and c over the lanes of equal bin b, which are consecutive lanes
// (b does not decrease along the warp); the last of them adds it to the
// block's histogram.  One shared-memory atomic per run of equal bins instead of
// one per element: shared FP64 atomics are compare-and-swap loops, and the
// lanes of a run all hit one address (256^3: 443 us with one atomic each).
__device__ __forceinline__ void add_runs(int b, double v, int c, int nbins, double* sv, int* sc) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int bo = __shfl_up_sync(0xffffffffu, b, o), co = __shfl_up_sync(0xffffffffu, c, o);
        const double vo = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o && bo == b) {
            v += vo;
            c += co;
        }
    }
    const int bn = __shfl_down_sync(0xffffffffu, b, 1);
    if ((lane == 31 || bn != b) && b < nbins) {
        atomicAdd(&sv[b], v);
        atomicAdd(&sc[b], c);
    }
}

// Shells of a 3-D array that is even along y and z up to mirror images: the
// images of a point at distances (x, y, z) from the origin, y <= ny/2 and
// z <= nz/2 (and x <= nx/2 where MIRROR_X), share its bin, so one lane sums
// them.  Warps walk rows of x.
//   K: half-spectrum modes (x = 0 .. nx/2, row length nx/2 + 1, modes with
//      0 < x < nx/2 stand for their conjugate partner too) into wavenumber
//      shells b = round(nmax * |(x/nx, y/ny, z/nz)|);
//   else: real-space separations (minimum image) into shells b = round(|r|).
template <class R, bool K>
__global__ void __launch_bounds__(kThreads) shell_kernel(const R* __restrict__ G, int nx, int ny, int nz, int nbins,
                                                         double* __restrict__ partials) {
    extern __shared__ double sh[];
    double* sv = sh;
    int* sc = reinterpret_cast<int*>(sh + nbins);
    for (int b = threadIdx.x; b < nbins; b += blockDim.x) {
        sv[b] = 0.0;
        sc[b] = 0;
    }
    __syncthreads();
    const int row = K ? nx / 2 + 1 : nx, hx = nx / 2 + 1, hy = ny / 2 + 1, hz = nz / 2 + 1;
    const double nmax = (double)max(nx, max(ny, nz));
    const int lane = threadIdx.x & 31, warps = (int)((gridDim.x * blockDim.x) >> 5);
    const int64_t rows = (int64_t)hy * hz;
    for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; r < rows; r += warps) {
        const int y = (int)(r % hy), z = (int)(r / hy);
        const int ny_im = (y == 0 || 2 * y == ny) ? 1 : 2, nz_im = (z == 0 || 2 * z == nz) ? 1 : 2;
        for (int x0 = 0; x0 < hx; x0 += 32) {
            const int x = x0 + lane;
            int b = nbins, cnt = 0;  // lanes past the row's end: no bin, last in the run order
            double v = 0.0;
            if (x < hx) {
                const bool edge = x == 0 || 2 * x == nx;
                if (K) {
                    const double fx = (double)x / nx, fy = (double)y / ny, fz = (double)z / nz;
                    b = (int)(nmax * sqrt(fx * fx + fy * fy + fz * fz) + 0.5);
                } else {
                    const double dx = x, dy = y, dz = z;
                    b = (int)(sqrt(dx * dx + dy * dy + dz * dz) + 0.5);
                }
                if (b < nbins) {
                    for (int iz = 0; iz < nz_im; ++iz)
                        for (int iy = 0; iy < ny_im; ++iy) {
                            const R* g = G + ((int64_t)(iz ? nz - z : z) * ny + (iy ? ny - y : y)) * row;
                            v += (double)g[x];
                            if (!K && !edge) v += (double)g[nx - x];
                        }
                    if (K && !edge) v *= 2.0;
                    cnt = nz_im * ny_im * (edge ? 1 : 2);
                } else {
                    b = nbins;
                }
            }
            add_runs(b, v, cnt, nbins, sv, sc);
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < nbins; b += blockDim.x) {
        partials[(size_t)b * gridDim.x + blockIdx.x] = sv[b];
        partials[((size_t)nbins + b) * gridDim.x + blockIdx.x] = (double)sc[b];
    }
}

// out[j] = sum over the blocks g of partials[j*G + g]: a warp per j, in a
// fixed order.
__global__ void __launch_bounds__(kThreads) fold_bins_kernel(const double* __restrict__ partials, int G, int n,
                                                             double* __restrict__ out) {
    const int j = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (j >= n) return;
    double acc = 0.0;
    for (int g = lane; g < G; g += 32) acc += partials[(size_t)j * G + g];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) out[j] = acc;
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Per block: sum |u| and sum |u|^2 into partials[q*G + block].
template <class R>
__global__ void __launch_bounds__(kThreads) speed_kernel(const R* __restrict__ u, int64_t V,
                                                         double* __restrict__ partials) {
    __shared__ double sh[2][kThreads / 32];
    double s1 = 0.0, s2 = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < V; i += (int64_t)gridDim.x * blockDim.x) {
        const double ux = u[i], uy = u[V + i], uz = u[2 * V + i];
        const double u2 = ux * ux + uy * uy + uz * uz;
        s1 += sqrt(u2);
        s2 += u2;
    }
    s1 = warp_sum_d(s1);
    s2 = warp_sum_d(s2);
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        sh[0][w] = s1;
        sh[1][w] = s2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int k = 0; k < kThreads / 32; ++k) {
            a += sh[0][k];
            b += sh[1][k];
        }
        partials[blockIdx.x] = a;
        partials[gridDim.x + blockIdx.x] = b;
    }
}

}  // namespace

struct Workspace {
    int nx = 0, ny = 0, nz = 0;
    int G = 0, Gs = 0;     // blocks of the shell and of the speed kernels
    bool dbl = false;
    int64_t V = 0, NC = 0;
    cufftHandle r2c = 0, c2r = 0;
    bool plans = false;
    void* A = nullptr;     // complex NC
    void* B = nullptr;     // complex NC (also the real C2R output)
    void* Rin = nullptr;   // real V: copy of a transformed component, if one is needed
    void* P = nullptr;     // real NC: accumulated power
    double* partials = nullptr;
    size_t partials_cap = 0;
    double* out = nullptr;  // device, 2 * kMaxBins
};

#define ST_CUDA(x)                                  \
    do {                                            \
        cudaError_t e_ = (x);                       \
        if (e_ != cudaSuccess) return (int)e_;      \
    } while (0)
#define ST_FFT(x)                                   \
    do {                                            \
        cufftResult r_ = (x);                       \
        if (r_ != CUFFT_SUCCESS) return 1000 + (int)r_; \
    } while (0)

Workspace* create(int nx, int ny, int nz, bool dbl, int num_sms) {
    Workspace* w = new Workspace;
    w->nx = nx;
    w->ny = ny;
    w->nz = nz;
    w->dbl = dbl;
    w->V = (int64_t)nx * ny * nz;
    w->NC = (int64_t)nz * ny * (nx / 2 + 1);
    w->G = 2 * std::max(1, num_sms);
    w->Gs = 8 * std::max(1, num_sms);
    return w;
}

void destroy(Workspace* w) {
    if (!w) return;
    if (w->plans) {
        cufftDestroy(w->r2c);
        cufftDestroy(w->c2r);
    }
    cudaFree(w->A);
    cudaFree(w->B);
    cudaFree(w->Rin);
    cudaFree(w->P);
    cudaFree(w->partials);
    cudaFree(w->out);
    delete w;
}

namespace {

size_t shell_smem(int nbins) { return (size_t)nbins * (sizeof(double) + sizeof(int)); }

int ensure(Workspace* w, int nbins, cudaStream_t st) {
    const size_t rb = w->dbl ? 8 : 4;
    if (!w->plans) {
        ST_FFT(cufftPlan3d(&w->r2c, w->nz, w->ny, w->nx, w->dbl ? CUFFT_D2Z : CUFFT_R2C));
        ST_FFT(cufftPlan3d(&w->c2r, w->nz, w->ny, w->nx, w->dbl ? CUFFT_Z2D : CUFFT_C2R));
        w->plans = true;
        ST_CUDA(cudaMalloc(&w->A, (size_t)w->NC * 2 * rb));
        ST_CUDA(cudaMalloc(&w->B, (size_t)w->NC * 2 * rb));
        ST_CUDA(cudaMalloc(&w->P, (size_t)w->NC * rb));
        ST_CUDA(cudaMalloc(&w->out, 2 * (size_t)kMaxBins * sizeof(double)));
        auto attr = [](auto k) {
            return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shell_smem(kMaxBins));
        };
        ST_CUDA(attr(shell_kernel<float, true>));
        ST_CUDA(attr(shell_kernel<double, true>));
        ST_CUDA(attr(shell_kernel<float, false>));
        ST_CUDA(attr(shell_kernel<double, false>));
    }
    ST_FFT(cufftSetStream(w->r2c, st));
    ST_FFT(cufftSetStream(w->c2r, st));
    const size_t need = std::max((size_t)w->G * 2 * nbins, (size_t)w->Gs * 2);
    if (need > w->partials_cap) {
        cudaFree(w->partials);
        w->partials = nullptr;
        ST_CUDA(cudaMalloc(&w->partials, need * sizeof(double)));
        w->partials_cap = need;
    }
    return 0;
}

// Forward transform of one component into dst.  The out-of-place
// real-to-complex transform leaves its input alone (of the out-of-place
// transforms only the complex-to-real one may overwrite it); a component whose
// address does not suit cuFFT's vector accesses (V not a multiple of 4) is
// copied first.
int forward(Workspace* w, const void* comp, void* dst, cudaStream_t st) {
    const size_t rb = w->dbl ? 8 : 4;
    if ((reinterpret_cast<uintptr_t>(comp) & 15) != 0) {
        if (!w->Rin) ST_CUDA(cudaMalloc(&w->Rin, (size_t)w->V * rb));
        ST_CUDA(cudaMemcpyAsync(w->Rin, comp, (size_t)w->V * rb, cudaMemcpyDeviceToDevice, st));
        comp = w->Rin;
    }
    if (w->dbl)
        ST_FFT(cufftExecD2Z(w->r2c, (cufftDoubleReal*)const_cast<void*>(comp), (cufftDoubleComplex*)dst));
    else
        ST_FFT(cufftExecR2C(w->r2c, (cufftReal*)const_cast<void*>(comp), (cufftComplex*)dst));
    return 0;
}

int power(Workspace* w, void* A, const void* B, int mode, cudaStream_t st) {
    const int grid = w->G * 4;
    if (w->dbl)
        power_kernel<double, cufftDoubleComplex><<<grid, kThreads, 0, st>>>(
            (cufftDoubleComplex*)A, (const cufftDoubleComplex*)B, (double*)w->P, w->NC, mode);
    else
        power_kernel<float, cufftComplex><<<grid, kThreads, 0, st>>>((cufftComplex*)A, (const cufftComplex*)B,
                                                                     (float*)w->P, w->NC, mode);
    ST_CUDA(cudaGetLastError());
    return 0;
}

int fold_to_host(Workspace* w, int nbins, double* v_host, double* c_host, cudaStream_t st) {
    const int n = 2 * nbins;
    fold_bins_kernel<<<(32 * n + kThreads - 1) / kThreads, kThreads, 0, st>>>(w->partials, w->G, n, w->out);
    ST_CUDA(cudaGetLastError());
    std::vector<double> tmp((size_t)n);
    ST_CUDA(cudaMemcpyAsync(tmp.data(), w->out, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost, st));
    ST_CUDA(cudaStreamSynchronize(st));
    std::memcpy(v_host, tmp.data(), (size_t)nbins * sizeof(double));
    if (c_host) std::memcpy(c_host, tmp.data() + nbins, (size_t)nbins * sizeof(double));
    return 0;
}

}  // namespace

int velocity_spectrum(Workspace* w, const void* u3, int nbins, double* E, double* counts, cudaStream_t st) {
    if (int r = ensure(w, nbins, st)) return r;
    const size_t rb = w->dbl ? 8 : 4;
    for (int c = 0; c < 3; ++c) {
        if (int r = forward(w, (const char*)u3 + (size_t)c * w->V * rb, w->A, st)) return r;
        if (int r = power(w, w->A, nullptr, c == 0 ? 0 : 1, st)) return r;
    }
    const size_t smem = shell_smem(nbins);
    if (w->dbl)
        shell_kernel<double, true><<<w->G, kThreads, smem, st>>>((const double*)w->P, w->nx, w->ny, w->nz, nbins,
                                                                 w->partials);
    else
        shell_kernel<float, true><<<w->G, kThreads, smem, st>>>((const float*)w->P, w->nx, w->ny, w->nz, nbins,
                                                                w->partials);
    ST_CUDA(cudaGetLastError());
    if (int r = fold_to_host(w, nbins, E, counts, st)) return r;
    const double norm = 0.5 / ((double)w->V * (double)w->V);
    for (int b = 0; b < nbins; ++b) E[b] *= norm;
    return 0;
}

int q_correlation(Workspace* w, const void* q5, int nbins, double* C, double* counts, cudaStream_t st) {
    if (int r = ensure(w, nbins, st)) return r;
    const size_t rb = w->dbl ? 8 : 4;
    auto comp = [&](int k) { return (const char*)q5 + (size_t)k * w->V * rb; };
    // Q:Q' = 2 xx xx' + 2 yy yy' + xx yy' + yy xx' + 2 (xy xy' + xz xz' + yz yz')
    // (qzz = -qxx - qyy), so its power is 2|X|^2 + 2|Y|^2 + 2 Re(X conj Y) + 2|.|^2 ...
    if (int r = forward(w, comp(0), w->A, st)) return r;
    if (int r = forward(w, comp(3), w->B, st)) return r;
    if (int r = power(w, w->A, w->B, 2, st)) return r;
    // the last component's pass leaves the power as a complex array (imaginary
    // part 0) in A; its inverse transform is the autocorrelation sum
    // V^2 <Q(x):Q(x+r)> at every separation r
    for (int k : {1, 2, 4}) {
        if (int r = forward(w, comp(k), w->A, st)) return r;
        if (int r = power(w, w->A, nullptr, k == 4 ? 4 : 3, st)) return r;
    }
    if (w->dbl)
        ST_FFT(cufftExecZ2D(w->c2r, (cufftDoubleComplex*)w->A, (cufftDoubleReal*)w->B));
    else
        ST_FFT(cufftExecC2R(w->c2r, (cufftComplex*)w->A, (cufftReal*)w->B));
    const size_t smem = shell_smem(nbins);
    if (w->dbl)
        shell_kernel<double, false><<<w->G, kThreads, smem, st>>>((const double*)w->B, w->nx, w->ny, w->nz, nbins,
                                                                  w->partials);
    else
        shell_kernel<float, false><<<w->G, kThreads, smem, st>>>((const float*)w->B, w->nx, w->ny, w->nz, nbins,
                                                                 w->partials);
    ST_CUDA(cudaGetLastError());
    std::vector<double> cnt((size_t)nbins);
    if (int r = fold_to_host(w, nbins, C, cnt.data(), st)) return r;
    // Shell means normalised by the r = 0 value (shell 0 holds r = 0 alone).
    const double g0 = cnt[0] > 0 ? C[0] / cnt[0] : 0.0;
    for (int b = 0; b < nbins; ++b) C[b] = (cnt[b] > 0 && g0 != 0.0) ? (C[b] / cnt[b]) / g0 : 0.0;
    if (counts) std::memcpy(counts, cnt.data(), (size_t)nbins * sizeof(double));
    return 0;
}

int speed_moments(Workspace* w, const void* u3, double* mean_speed, double* mean_speed2, cudaStream_t st) {
    if (int r = ensure(w, 2, st)) return r;
    if (w->dbl)
        speed_kernel<double><<<w->Gs, kThreads, 0, st>>>((const double*)u3, w->V, w->partials);
    else
        speed_kernel<float><<<w->Gs, kThreads, 0, st>>>((const float*)u3, w->V, w->partials);
    ST_CUDA(cudaGetLastError());
    fold_bins_kernel<<<1, kThreads, 0, st>>>(w->partials, w->Gs, 2, w->out);
    ST_CUDA(cudaGetLastError());
    double r[2];
    ST_CUDA(cudaMemcpyAsync(r, w->out, sizeof(r), cudaMemcpyDeviceToHost, st));
    ST_CUDA(cudaStreamSynchronize(st));
    *mean_speed = r[0] / (double)w->V;
    *mean_speed2 = r[1] / (double)w->V;
    return 0;
}

bool is_nomem(int code) {
    return code == (int)cudaErrorMemoryAllocation || code == 1000 + (int)CUFFT_ALLOC_FAILED;
}

const char* err_string(int code) {
    if (code >= 1000) {
        switch (code - 1000) {
            case CUFFT_ALLOC_FAILED: return "cuFFT: allocation failed";
            case CUFFT_INVALID_VALUE: return "cuFFT: invalid value";
            case CUFFT_INVALID_SIZE: return "cuFFT: invalid size";
            case CUFFT_EXEC_FAILED: return "cuFFT: execution failed";
            case CUFFT_SETUP_FAILED: return "cuFFT: setup failed";
            default: return "cuFFT error";
        }
    }
    return cudaGetErrorString((cudaError_t)code);
}

}  // namespace stats
}  // namespace lbman
