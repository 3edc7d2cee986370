// reduce.cuh -- diagnostic reductions on the device: SimIO::Log's sums
// (src/sim_io.cc:83-108), TotalNematicFreeEnergy (src/analysis_fields.h:39-72),
// QtensorToOrderDirector (src/analysis_fields.cc:59-93) and the plaquette
// sign-flip flags of DefectFinder::ComputeWindingNumbers
// (src/analysis/defect_finder.tpp:13-165).
//
// Accumulation is FP64 whatever the field precision.  Pass 1: grid-stride
// loop, warp-shuffle then shared-memory reduction, one partial per block
// (partials[q*G + block]).  Pass 2: one block folds the partials in a fixed
// order, so results are deterministic run to run.
#pragma once

#include "common.cuh"

#include <algorithm>

namespace lbman {

constexpr int kRedThreads = 256;
constexpr int kFlowQ = 8;  // mass px py pz ke e1 e2 | umax2

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

// Block reduction of NQ values (the last NMAX of them by max).  Thread 0
// writes partials[q*gridDim.x + blockIdx.x].
template <int NQ, int NMAX>
__device__ __forceinline__ void block_reduce_store(double (&v)[NQ], double* partials) {
    __shared__ double sh[NQ][kRedThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const double r = q < NQ - NMAX ? warp_sum(v[q]) : warp_max(v[q]);
        if (lane == 0) sh[q][warp] = r;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            double r = lane < (int)(blockDim.x >> 5) ? sh[q][lane] : (q < NQ - NMAX ? 0.0 : -1.0);
            r = q < NQ - NMAX ? warp_sum(r) : warp_max(r);
            if (lane == 0) partials[(size_t)q * gridDim.x + blockIdx.x] = r;
        }
    }
}

__device__ __forceinline__ void flow_cell(double (&v)[kFlowQ], double r, double ux, double uy, double uz, double px,
                                          double py, double pz) {
    v[0] += r;
    v[1] += r * ux;
    v[2] += r * uy;
    v[3] += r * uz;
    const double u2 = ux * ux + uy * uy + uz * uz;
    v[4] += 0.5 * r * u2;
    v[5] += (ux - px) * (ux - px) + (uy - py) * (uy - py) + (uz - pz) * (uz - pz);
    v[6] += u2;
    v[7] = fmax(v[7], u2);
}

// Memory bound (10 words per cell): two cells per thread and turn, all their
// loads issued before the first use.  256^3 FP32: 111 us; one cell at a time
// 161-191 us, four neighbouring cells as 16-byte accesses 424 us (the lanes'
// accesses to seven arrays at that stride collide in the cache).
template <class R>
__global__ void __launch_bounds__(kRedThreads) flow_reduce_kernel(SimParams P, const R* __restrict__ rho,
                                                                  const R* __restrict__ u,
                                                                  R* __restrict__ upast,
                                                                  double* __restrict__ partials) {
    const int64_t V = P.V, nt = (int64_t)gridDim.x * blockDim.x;
    double v[kFlowQ] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int64_t c = P.c0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < P.c1; c += 2 * nt) {
        R r[2], a[2][3], b[2][3];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int64_t d = c + i * nt;
            if (d < P.c1) {
                r[i] = rho[d];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    a[i][k] = u[k * V + d];
                    b[i][k] = upast[k * V + d];
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int64_t d = c + i * nt;
            if (d < P.c1) {
                flow_cell(v, (double)r[i], (double)a[i][0], (double)a[i][1], (double)a[i][2], (double)b[i][0],
                          (double)b[i][1], (double)b[i][2]);
#pragma unroll
                for (int k = 0; k < 3; ++k) upast[k * V + d] = a[i][k];
            }
        }
    }
    block_reduce_store<kFlowQ, 1>(v, partials);
}

// Planes per work item of the z-marching diagnostics (one thread per column of
// an x-y tile): as many as leave 8 items for each of the part's 148 SMs, between
// 2 and 32 -- a longer march re-reads less, a shorter one fills the chip.
// Defects, 20x100x100 FP64: 18 us at 2 planes, 70 us at 32; 256^3 FP32: 610 us
// at 2, 472 us at 32.  Energy: 13 / 31 us and 337 / 252 us.
inline int diag_planes(int64_t tiles, int nz) {
    const int64_t chunks = (8 * 148 + tiles - 1) / tiles;
    return (int)std::max<int64_t>(2, std::min<int64_t>(32, (nz + chunks - 1) / chunks));
}

// Index of the neighbour a + s under the QXoff clamp / wrap of one axis.
__device__ __forceinline__ int qx_off(int a, int n, int per_lo, int per_hi) {
    if (a < 0) return per_lo ? a + n : 0;
    if (a >= n) return per_hi ? a - n : n - 1;
    return a;
}

// NematicFreeEnergyDensity with the QXoff-clamped 7-point Laplacian, in FP64.
// FP32 fields: a value is converted once -- each thread converts its own
// column, keeps three planes of it in registers and shares the current plane
// through shared memory -- because the conversions (a fraction of the FP64
// rate) were what bounded the one-thread-per-cell form, with 35 per cell.  The
// next plane's values are loaded while this one is worked on.  256^3 FP32:
// 331 us one thread per cell, 252 us now at 3 blocks per SM (293 at 2, 294 at
// 4, which spills); FP64, which converts nothing: 343-352 us at 2 blocks, 369 at 3.
// Neither HBM (1.4 TB/s) nor the FP64 pipe (29% active) bounds it: issue slots are
// 55% used, at 23 warps per SM and one barrier per plane.
constexpr int kEnX = 32, kEnY = 8;
static_assert(kEnX * kEnY == kRedThreads, "one thread per column of a tile");
template <class R>
__global__ void __launch_bounds__(kRedThreads, sizeof(R) == 4 ? 3 : 2) energy_reduce_kernel(const __grid_constant__ SimParams P,
                                                                    int zc, const R* __restrict__ q,
                                                                    double* __restrict__ partials) {
    constexpr int SX = kEnX + 2, SY = kEnY + 2;
    __shared__ double sh[2][5][SY][SX];
    const int64_t V = P.V;
    const int nx = P.nx, ny = P.ny, nz = P.nz;
    double v[1] = {0.0};
    int b = 0;
    const int gx = (nx + kEnX - 1) / kEnX, gy = (ny + kEnY - 1) / kEnY, gz = (P.zhi - P.zlo + zc - 1) / zc;
    const int lx = threadIdx.x % kEnX, ly = threadIdx.x / kEnX;
    // this thread's halo point of a plane (threads 0 .. 2 (kEnX + kEnY) - 1)
    const int h = threadIdx.x;
    const bool halo = h < 2 * (kEnX + kEnY);
    const int hx = h < 2 * kEnX ? h % kEnX + 1 : (h - 2 * kEnX < kEnY ? 0 : SX - 1);
    const int hy = h < 2 * kEnX ? (h < kEnX ? 0 : SY - 1) : (h - 2 * kEnX) % kEnY + 1;
    for (int item = blockIdx.x; item < gx * gy * gz; item += gridDim.x) {
        const int x0 = item % gx * kEnX, y0 = item / gx % gy * kEnY, z0 = P.zlo + item / (gx * gy) * zc;
        const int z1 = min(z0 + zc, P.zhi);
        const int x = x0 + lx, y = y0 + ly;
        const bool live = x < nx && y < ny;
        const int64_t col = (int64_t)min(y, ny - 1) * nx + min(x, nx - 1);
        const int64_t hcol = (int64_t)qx_off(min(y0 + hy - 1, ny), ny, P.qper[2], P.qper[3]) * nx +
                             qx_off(min(x0 + hx - 1, nx), nx, P.qper[0], P.qper[1]);
        const R* const qx = q + col;
        const R* const qh = q + hcol;
        double qm[5], qc[5];
        R rp[5], rh[5];  // plane z + 1 of the column, plane z of the halo point
        const int64_t zm0 = (int64_t)qx_off(z0 - 1, nz, P.qper[4], P.qper[5]) * P.nxy;
        const int64_t zp0 = (int64_t)qx_off(z0 + 1, nz, P.qper[4], P.qper[5]) * P.nxy;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            qm[k] = (double)qx[k * V + zm0];
            qc[k] = (double)qx[k * V + (int64_t)z0 * P.nxy];
            rp[k] = qx[k * V + zp0];
            rh[k] = qh[k * V + (int64_t)z0 * P.nxy];
        }
        for (int z = z0; z < z1; ++z) {
            b ^= 1;
            double qp[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                sh[b][k][ly + 1][lx + 1] = qc[k];
                if (halo) sh[b][k][hy][hx] = (double)rh[k];
                qp[k] = (double)rp[k];
            }
            __syncthreads();  // the other buffer's readers are at most one plane behind
            if (z + 1 < z1) {
                const int64_t zn = (int64_t)qx_off(z + 2, nz, P.qper[4], P.qper[5]) * P.nxy;
#pragma unroll
                for (int k = 0; k < 5; ++k) {
                    rp[k] = qx[k * V + zn];
                    rh[k] = qh[k * V + (int64_t)(z + 1) * P.nxy];
                }
            }
            if (live) {
                // the neighbour beyond a partial tile's last cell comes from
                // global memory (its shared slot holds a column outside the box)
                double l[5];
#pragma unroll
                for (int k = 0; k < 5; ++k) {
                    const R* a = q + k * V + (int64_t)z * P.nxy;
                    const double xp = (x == nx - 1 && lx != kEnX - 1)
                                          ? (double)a[(int64_t)y * nx + qx_off(nx, nx, P.qper[0], P.qper[1])]
                                          : sh[b][k][ly + 1][lx + 2];
                    const double yp = (y == ny - 1 && ly != kEnY - 1)
                                          ? (double)a[(int64_t)qx_off(ny, ny, P.qper[2], P.qper[3]) * nx + x]
                                          : sh[b][k][ly + 2][lx + 1];
                    l[k] = xp + sh[b][k][ly + 1][lx] + yp + sh[b][k][ly][lx + 1] + qp[k] + qm[k] - 6.0 * qc[k];
                }
                const double Qxx = qc[0], Qxy = qc[1], Qxz = qc[2], Qyy = qc[3], Qyz = qc[4];
                const double half = (Qxx * Qxx + Qxx * Qyy + Qyy * Qyy + Qxy * Qxy + Qxz * Qxz + Qyz * Qyz);
                const double TrQ2 = 2.0 * half;
                const double k13 = 1.0 / 3.0;
                const double Q2_xx = Qxx * Qxx + Qxy * Qxy + Qxz * Qxz - k13 * TrQ2;
                const double Q2_xy = Qxx * Qxy + Qxy * Qyy + Qxz * Qyz;
                const double Q2_xz = Qxy * Qyz - Qxz * Qyy;
                const double Q2_yy = Qxy * Qxy + Qyy * Qyy + Qyz * Qyz - k13 * TrQ2;
                const double Q2_yz = Qxy * Qxz - Qyz * Qxx;
                const double TrQ3 = 2.0 * Qxx * Q2_xx + 2.0 * Qyy * Q2_yy + Qxx * Q2_yy + Qyy * Q2_xx +
                                    2.0 * (Qxy * Q2_xy + Qxz * Q2_xz + Qyz * Q2_yz);
                const double QlQ = 2.0 * Qxx * l[0] + 2.0 * Qyy * l[3] + Qxx * l[3] + Qyy * l[0] +
                                   2.0 * (Qxy * l[1] + Qxz * l[2] + Qyz * l[4]);
                v[0] += 0.5 * P.A * TrQ2 + (P.B / 3.0) * TrQ3 + 0.25 * P.C * TrQ2 * TrQ2 - 0.5 * P.L * QlQ;
            }
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                qm[k] = qc[k];
                qc[k] = qp[k];
            }
        }
    }
    block_reduce_store<1, 0>(v, partials);
}

// Director n of a cell (closed form, no diagonalisation), in FP64, rounded to
// the field's precision.
template <class R>
__device__ __forceinline__ void director(double Qxx, double Qxy, double Qxz, double Qyy, double Qyz, R n[3]) {
    const double pp = (Qxx * Qxx + Qxx * Qyy + Qyy * Qyy + Qxy * Qxy + Qxz * Qxz + Qyz * Qyz);
    const double qq = (-(Qxx + Qyy) * (Qxx * Qyy - Qxy * Qxy) - Qyy * Qxz * Qxz - Qxx * Qyz * Qyz +
                       2 * Qxy * Qxz * Qyz);
    const double r = 2.0 * sqrt(pp / 3.0);
    double arg = 4 * qq / (r * r * r);
    arg = arg < -1.0 ? -1.0 : (1.0 < arg ? 1.0 : arg);
    const double S = r * cos(1.0 / 3.0 * acos(arg));
    double nx_ = Qxz * (Qyy - S) - Qxy * Qyz;
    double ny_ = Qyz * (Qxx - S) - Qxy * Qxz;
    double nz_ = Qxy * Qxy - (Qxx - S) * (Qyy - S);
    const double ninv = 1.0 / sqrt(nx_ * nx_ + ny_ * ny_ + nz_ * nz_);
    n[0] = (R)(nx_ * ninv);
    n[1] = (R)(ny_ * ninv);
    n[2] = (R)(nz_ * ninv);
}

// Is a.b <= 0, with b negated if flip: decided in FP64.  For FP32 directors an
// FP32 evaluation decides first: three products of components of at most 1 in
// magnitude sum with an error below 3e-7, so beyond 1e-6 its sign is the FP64
// one (NaN takes the FP64 branch).
__device__ __forceinline__ bool dot_nonpositive(const double a[3], const double b[3], bool flip) {
    const double d = a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
    return (flip ? -d : d) <= 0.0;
}
__device__ __forceinline__ bool dot_nonpositive(const float a[3], const float b[3], bool flip) {
    const float d = fmaf(a[2], b[2], fmaf(a[1], b[1], a[0] * b[0]));
    if (fabsf(d) > 1e-6f) return flip ? d > 0.0f : d < 0.0f;
    const double e = (double)a[0] * b[0] + (double)a[1] * b[1] + (double)a[2] * b[2];
    return (flip ? -e : e) <= 0.0;
}
// Do the directors of a plaquette, each made to point along the one before,
// end up against the first (src/analysis/defect_finder.tpp)?  The signs of the
// second to fourth are kept as flips.
template <class R>
__device__ __forceinline__ bool plaquette_flip(const R d1[3], const R d2[3], const R d3[3], const R d4[3]) {
    const bool f2 = dot_nonpositive(d1, d2, false);
    const bool f3 = dot_nonpositive(d2, d3, f2);
    const bool f4 = dot_nonpositive(d3, d4, f3);
    return dot_nonpositive(d4, d1, f4);
}

// Plaquette sign-flip flags of the three face families in one z march: a
// thread evaluates the director of one column, planes z and z - 1 meet in shared
// memory, and the threads of the tile's first kDefX x kDefY columns test the
// three plaquettes of their cell.  Bound by the director's FP64 arithmetic
// (each is formed 1.1 times), where a director pass and a pass over its 24-byte
// records took 567 us for 256^3 FP32.  The periodic seam faces are not visited,
// as in the reference.
// Block (bx, by, bz) of tiles and z chunks is one of the launch's x dimension:
// long or tall boxes have more than the 65535 the others take.
//   count: receives the number of flagged plaquettes (added atomically);
//   flags: if not null, the flags in the reference's DefectFields layout
//   (src/analysis/defect_fields.h:16-29): def_x nx*(ny-1)*(nz-1), then def_y
//   (nx-1)*ny*(nz-1), then def_z (nx-1)*(ny-1)*nz, each x fastest.
constexpr int kDefTX = 32, kDefTY = 16, kDefX = kDefTX - 1, kDefY = kDefTY - 1, kDefThreads = kDefTX * kDefTY;
template <class R>
__global__ void __launch_bounds__(kDefThreads) defect_kernel(const __grid_constant__ SimParams P, int zc,
                                                             const R* __restrict__ q, uint8_t* __restrict__ flags,
                                                             unsigned long long* __restrict__ count) {
    __shared__ R sh[2][3][kDefTY][kDefTX];
    __shared__ int total;
    const int64_t V = P.V;
    const int nx = P.nx, ny = P.ny, nz = P.nz;
    const int64_t nfx = (int64_t)nx * (ny - 1) * (nz - 1), nfy = (int64_t)(nx - 1) * ny * (nz - 1);
    const int lx = threadIdx.x % kDefTX, ly = threadIdx.x / kDefTX;
    const int gx = (nx + kDefX - 1) / kDefX, gy = (ny + kDefY - 1) / kDefY;
    const int bx = blockIdx.x % gx, by = blockIdx.x / gx % gy, bz = blockIdx.x / gx / gy;
    const int x = bx * kDefX + lx, y = by * kDefY + ly;
    const int z0 = bz * zc, z1 = min(z0 + zc, nz);  // def_z planes of this block
    const bool in = x < nx && y < ny;
    const bool own = in && lx < kDefX && ly < kDefY;
    const int64_t col = (int64_t)y * nx + x;
    if (threadIdx.x == 0) total = 0;
    auto at = [&](int b, int dx, int dy, R d[3]) {
#pragma unroll
        for (int k = 0; k < 3; ++k) d[k] = sh[b][k][ly + dy][lx + dx];
    };
    int n = 0;
    for (int z = z0; z <= min(z1, nz - 1); ++z) {
        const int b = z & 1;
        if (in) {
            const R* a = q + (int64_t)z * P.nxy + col;
            R d[3];
            director<R>((double)a[0], (double)a[V], (double)a[2 * V], (double)a[3 * V], (double)a[4 * V], d);
#pragma unroll
            for (int k = 0; k < 3; ++k) sh[b][k][ly][lx] = d[k];
        }
        __syncthreads();
        if (own) {
            R d00[3], d10[3], d01[3];
            at(b, 0, 0, d00);
            if (x < nx - 1) at(b, 1, 0, d10);
            if (y < ny - 1) at(b, 0, 1, d01);
            if (z < z1 && x < nx - 1 && y < ny - 1) {  // def_z of plane z
                R d11[3];
                at(b, 1, 1, d11);
                const bool f = plaquette_flip<R>(d00, d10, d11, d01);
                n += f;
                if (flags) flags[nfx + nfy + ((int64_t)z * (ny - 1) + y) * (nx - 1) + x] = f;
            }
            if (z > z0) {  // def_x, def_y between the planes z - 1 and z
                R p00[3];
                at(b ^ 1, 0, 0, p00);
                if (y < ny - 1) {
                    R p01[3];
                    at(b ^ 1, 0, 1, p01);
                    const bool f = plaquette_flip<R>(p00, p01, d01, d00);
                    n += f;
                    if (flags) flags[((int64_t)(z - 1) * (ny - 1) + y) * nx + x] = f;
                }
                if (x < nx - 1) {
                    R p10[3];
                    at(b ^ 1, 1, 0, p10);
                    const bool f = plaquette_flip<R>(p00, p10, d10, d00);
                    n += f;
                    if (flags) flags[nfx + ((int64_t)(z - 1) * ny + y) * (nx - 1) + x] = f;
                }
            }
        }
        __syncthreads();  // plane z - 1's slot takes plane z + 1
    }
    for (int o = 16; o > 0; o >>= 1) n += __shfl_down_sync(0xffffffffu, n, o);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(&total, n);
    __syncthreads();
    if (threadIdx.x == 0 && total) atomicAdd(count, (unsigned long long)total);
}

// Pass 2: fold G partials of NQ quantities (the last nmax by max) in order.
static __global__ void __launch_bounds__(1024) fold_partials_kernel(const double* __restrict__ partials, int G,
                                                             int nq, int nmax, double* __restrict__ out) {
    __shared__ double sh[32];
    for (int q = 0; q < nq; ++q) {
        const bool is_max = q >= nq - nmax;
        double acc = is_max ? -1.0 : 0.0;
        for (int b = threadIdx.x; b < G; b += blockDim.x) {
            const double x = partials[(size_t)q * G + b];
            acc = is_max ? fmax(acc, x) : acc + x;
        }
        acc = is_max ? warp_max(acc) : warp_sum(acc);
        if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
        __syncthreads();
        if (threadIdx.x < 32) {
            double r = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : (is_max ? -1.0 : 0.0);
            r = is_max ? warp_max(r) : warp_sum(r);
            if (threadIdx.x == 0) out[q] = r;
        }
        __syncthreads();
    }
}

}  // namespace lbman
