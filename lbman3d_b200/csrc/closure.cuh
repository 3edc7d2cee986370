// closure.cuh -- kernels of the learned closure: a 4-layer 3x3x3 periodic
// convolutional network (9 -> 32 -> 32 -> 32 -> 8 channels, GELU after the
// first three layers) on a coarse grid, with BF16 operands on the tcgen05
// tensor cores and FP32 accumulation in TMEM.  No counterpart in the
// reference.
//
// Activations are channel-last BF16, act[cell][C] with C = 16 (the 9 input
// features, zero padded) or 32; the last layer's 8 outputs are padded to 16.
// A convolution is an implicit GEMM: for a tile of 128 cells (M) and each of
// the 27 taps, the 128 x CIN neighbour rows are gathered into shared memory
// (K-major) and multiplied by that tap's CIN x COUT weights (N = COUT), all
// 27 taps accumulating into one TMEM accumulator.  Two A stages let the
// gather of tap t+1 overlap the MMAs of tap t.  The backward data pass is
// the same kernel run with the transposed, tap-reversed weight image; the
// weight gradient is a GEMM over cells (K) with M = (tap, ci) rows and
// MN-major operands taken straight from the channel-last activations.
//
// Tap index: tap = (dz+1)*9 + (dy+1)*3 + (dx+1); output cell c reads input
// cell c + (dx, dy, dz) with periodic wrap on every axis.
//
// Waits: every wait for MMA completion that the pipeline needs to go on
// polls at most wait_limit times (a kernel argument; tc::kWaitLimit unless
// the caller lowered it).  A wait that gives up sets *err, the whole CTA
// leaves its tile loop together (__syncthreads_or), and the drain waits --
// always with the full tc::kWaitLimit, because the tensor core must finish
// every MMA it was given before the CTA frees its TMEM -- end the kernel.
#pragma once

#include <cuda_bf16.h>
#include <stdint.h>

#include "pdl.cuh"
#include "tc.cuh"

namespace lbman {
namespace cl {

constexpr int kTileM = 128;
constexpr int kThreads = 128;
constexpr int kOutChannels = 8;  // of the network; its output is channel-major, [8][V]
constexpr int kStages = 4;  // A-operand stages of the convolution pipeline

struct Grid3 {
    int nx, ny, nz;
    int64_t V;
};

__device__ __forceinline__ int wrapi(int a, int n) { return a < 0 ? a + n : (a >= n ? a - n : a); }

__device__ __forceinline__ int64_t neighbour(const Grid3& g, int x, int y, int z, int tap) {
    const int dx = tap % 3 - 1, dy = (tap / 3) % 3 - 1, dz = tap / 9 - 1;
    return ((int64_t)wrapi(z + dz, g.nz) * g.ny + wrapi(y + dy, g.ny)) * g.nx + wrapi(x + dx, g.nx);
}

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
    const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
    return cdf + x * pdf;
}

// Byte size of the B image of one convolution: 27 taps x CIN/16 k-steps of
// COUT x 16 K-major BF16 blocks (core matrices: n-group stride 256, k-group 128).
__host__ __device__ constexpr int bimg_bytes(int cin, int cout) { return 27 * (cin / 16) * cout * 32; }

// Byte offset in the B image of the COUT x 16 block of (dy, dx) index yx, k-step
// kb and dz: the three dz of a (yx, kb) are consecutive, +1 first.
__host__ __device__ constexpr int bimg_off(int cin, int cout, int yx, int kb, int dz) {
    return ((yx * (cin / 16) + kb) * 3 + (1 - dz)) * cout * 32;
}

enum ConvMode : int {
    kFwdHidden = 0,  // + bias, store pre (BF16) and GELU(pre) (BF16)
    kFwdLast = 1,    // + bias, store FP32 channel-major
    kBwdData = 2     // times GELU'(pre of the layer below), store BF16
};

// Halo staging applies when a 128-cell tile is R = 128/nx whole x rows of
// one z plane: then the tile's input neighbourhood (3 planes x R+2 rows x nx
// cells) is copied into shared memory once per tile and the 27 tap operands
// are built from it, instead of 27 gathers from L2.
__host__ __device__ inline bool halo_ok(int nx, int ny) {
    return nx <= kTileM && kTileM % nx == 0 && ((int64_t)nx * ny) % kTileM == 0;
}
__host__ __device__ inline int halo_bytes(int nx, int cin) { return 3 * (kTileM / nx + 2) * nx * cin * 2; }

// One persistent CTA walks 128-cell tiles.  Smem: B image, kStages A stages
// of CIN/16 x 4 KB, then (halo != 0) the staged neighbourhood.  The operand
// of tap k goes to stage k % kStages once the MMAs that last read that stage
// have completed, so operand copies run up to kStages - 1 taps ahead of the
// tensor core.  Halo units of
// 16 bytes are stored at cell * (CIN/8) + (q ^ (cell & (CIN/8 - 1))), an XOR
// swizzle that spreads a warp's reads of one q over the banks.
template <int CIN, int COUT, int MODE>
__global__ void __launch_bounds__(kThreads) conv_kernel(Grid3 g, const __nv_bfloat16* __restrict__ in,
                                                        const uint4* __restrict__ bimg, const float* __restrict__ bias,
                                                        const __nv_bfloat16* __restrict__ pre_below,
                                                        __nv_bfloat16* __restrict__ out_pre,
                                                        __nv_bfloat16* __restrict__ out_bf, float* __restrict__ out_f,
                                                        int halo, int* __restrict__ err,
        uint32_t wait_limit) {
    constexpr int KS = CIN / 16;                 // k-steps per tap
    constexpr int BBYTES = bimg_bytes(CIN, COUT);
    constexpr int ABYTES = KS * 4096;            // one A stage
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ uint64_t bar[kStages];
    __shared__ uint32_t tslot;
    constexpr int QU = CIN / 8;                  // 16-byte units per cell
    unsigned char* Bs = sm;
    unsigned char* As = sm + BBYTES;
    uint4* Hs = reinterpret_cast<uint4*>(sm + BBYTES + kStages * ABYTES);
    const int t = threadIdx.x;
    const int R = kTileM / g.nx;                 // rows per tile (halo path)

    for (int i = t; i < BBYTES / 16; i += kThreads) reinterpret_cast<uint4*>(Bs)[i] = bimg[i];
    if (t == 0) {
        for (int k = 0; k < kStages; ++k) tc::mbar_init(&bar[k], 1);
        tc::mbar_fence_init();
    }
    if (t < 32) tc::tmem_alloc(&tslot, 32);
    tc::fence_smem_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tslot;
    const uint32_t idesc = tc::idesc_bf16(kTileM, COUT, 0, 0);
    const uint32_t a0 = tc::smem_addr(As), b0 = tc::smem_addr(Bs);
    uint32_t uses[kStages] = {};  // commits issued per A stage (same in every thread)
    int kt = 0;                     // taps issued so far by this CTA
    int last_s = 0;
    bool ok = true;

    const int64_t ntiles = (g.V + kTileM - 1) / kTileM;
    for (int64_t tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        const int64_t c = tile * kTileM + t;
        const bool live = c < g.V;
        const int64_t cc = live ? c : 0;
        const int x = (int)(cc % g.nx), y = (int)((cc / g.nx) % g.ny), z = (int)(cc / ((int64_t)g.nx * g.ny));
        if (halo) {
            // planes z0-1..z0+1, rows y0-1..y0+R of the tile's plane
            const int64_t c0 = tile * kTileM;
            const int z0 = (int)(c0 / ((int64_t)g.nx * g.ny)), y0 = (int)((c0 / g.nx) % g.ny);
            const int nunits = 3 * (R + 2) * g.nx * QU;
            for (int i = t; i < nunits; i += kThreads) {
                const int q = i % QU, cell = i / QU;
                const int hx = cell % g.nx, hr = (cell / g.nx) % (R + 2), hz = cell / (g.nx * (R + 2));
                const int64_t src = ((int64_t)wrapi(z0 - 1 + hz, g.nz) * g.ny + wrapi(y0 - 1 + hr, g.ny)) * g.nx + hx;
                const uint4* gp = reinterpret_cast<const uint4*>(in + src * CIN) + q;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                                 tc::smem_addr(Hs + cell * QU + (q ^ (cell & (QU - 1))))),
                             "l"(gp));
            }
            asm volatile("cp.async.wait_all;\n" ::: "memory");
            __syncthreads();
        }
        for (int tap = 0; tap < 27; ++tap, ++kt) {
            const int s = kt % kStages;
            // stage s is free once the MMAs that read it last have completed
            bool lost = uses[s] > 0 && !tc::mbar_wait(&bar[s], (uses[s] - 1) & 1, err, wait_limit);
            if (__syncthreads_or(lost)) {
                ok = false;
                break;
            }
            // this row's CIN channels of the neighbour into stage s
            unsigned char* dst = As + s * ABYTES + (t / 8) * 256 + (t % 8) * 16;
            if (halo) {
                const int dx = tap % 3 - 1, dy = (tap / 3) % 3 - 1, dz = tap / 9 - 1;
                const int hx = wrapi(t % g.nx + dx, g.nx), hr = t / g.nx + 1 + dy;
                const int cell = ((1 + dz) * (R + 2) + hr) * g.nx + hx;
#pragma unroll
                for (int q = 0; q < QU; ++q)
                    *reinterpret_cast<uint4*>(dst + (q / 2) * 4096 + (q % 2) * 128) =
                        Hs[cell * QU + (q ^ (cell & (QU - 1)))];
            } else {
                const uint4* src = reinterpret_cast<const uint4*>(in + neighbour(g, x, y, z, tap) * CIN);
#pragma unroll
                for (int q = 0; q < QU; ++q)
                    *reinterpret_cast<uint4*>(dst + (q / 2) * 4096 + (q % 2) * 128) = src[q];
            }
            tc::fence_smem_async();
            tc::fence_before_sync();
            __syncthreads();
            tc::fence_after_sync();
            if (t == 0) {
#pragma unroll
                for (int kb = 0; kb < KS; ++kb) {
                    const uint64_t da = tc::smem_desc(a0 + s * ABYTES + kb * 4096, 128, 256);
                    const uint64_t db = tc::smem_desc(b0 + bimg_off(CIN, COUT, tap % 9, kb, tap / 9 - 1), 128, 256);
                    tc::mma_bf16(tmem, da, db, idesc, (tap > 0 || kb > 0) ? 1u : 0u);
                }
                tc::mma_commit(&bar[s]);
            }
            ++uses[s];
            last_s = s;
        }
        if (!ok) break;
        // the tile's last commit covers every MMA issued before it
        const bool lost = !tc::mbar_wait(&bar[last_s], (uses[last_s] - 1) & 1, err, wait_limit);
        if (__syncthreads_or(lost)) {
            ok = false;
            break;
        }
        tc::fence_after_sync();
        const int w = t >> 5;
        float acc[COUT];
#pragma unroll
        for (int c0 = 0; c0 < COUT; c0 += 16) tc::tmem_ld16(tmem + ((uint32_t)(32 * w) << 16) + (uint32_t)c0, acc + c0);
        if (live) {
            if constexpr (MODE == kFwdHidden) {
                __align__(16) __nv_bfloat16 pb[COUT], ab[COUT];
#pragma unroll
                for (int j = 0; j < COUT; ++j) {
                    const float p = acc[j] + bias[j];
                    pb[j] = __float2bfloat16(p);
                    ab[j] = __float2bfloat16(gelu(p));
                }
#pragma unroll
                for (int q = 0; q < COUT / 8; ++q) {
                    reinterpret_cast<uint4*>(out_pre + c * COUT)[q] = reinterpret_cast<const uint4*>(pb)[q];
                    reinterpret_cast<uint4*>(out_bf + c * COUT)[q] = reinterpret_cast<const uint4*>(ab)[q];
                }
            } else if constexpr (MODE == kFwdLast) {
#pragma unroll
                for (int j = 0; j < kOutChannels; ++j) out_f[j * g.V + c] = acc[j] + bias[j];
            } else {
                __align__(16) __nv_bfloat16 pre[COUT], gb[COUT];
#pragma unroll
                for (int q = 0; q < COUT / 8; ++q)
                    reinterpret_cast<uint4*>(pre)[q] = reinterpret_cast<const uint4*>(pre_below + c * COUT)[q];
#pragma unroll
                for (int j = 0; j < COUT; ++j) gb[j] = __float2bfloat16(acc[j] * gelu_grad(__bfloat162float(pre[j])));
#pragma unroll
                for (int q = 0; q < COUT / 8; ++q)
                    reinterpret_cast<uint4*>(out_bf + c * COUT)[q] = reinterpret_cast<const uint4*>(gb)[q];
            }
        }
        tc::fence_before_sync();
        __syncthreads();  // TMEM reads done before the next tile's first MMA
        tc::fence_after_sync();
    }
    // drain: never leave with MMAs in flight on our TMEM
    if (t == 0) {
        for (int s = 0; s < kStages; ++s)
            if (uses[s] > 0) tc::mbar_wait(&bar[s], (uses[s] - 1) & 1, err);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (t < 32) tc::tmem_dealloc(tmem, 32);
}

// ---- descriptor-halo convolution, z-marching ---------------------------------
// Tile = 8 x-cells by 16 y-rows of one z plane (128 cells, M row m = 8*dy_row
// + dx_cell).  A CTA takes a column of tiles (the same 8 x 16 block of every
// plane of a z range) and marches it in z.  The column's neighbourhood is
// staged plane by plane (10 x 18 cells per plane) in a ring of 3 plane slots,
// as 16-byte units, one block per 8-channel group:
//   unit(slot, kg, hy, hx) at slot*SLOT + (kg*18 + hy)*10 + hx,
// which makes the A operand of every (dx, dy) a K-major view of a slot: rows
// of a core matrix are 8 consecutive x cells (16 bytes apart), the next y row
// is SBO = 160 bytes on, the next 8 channels LBO = 2880 bytes on, and (dx, dy)
// only moves the start address.
//
// A staged plane is multiplied once, by the weights of all three dz at once:
// N = 3 COUT columns, the accumulators of the output planes z - 1, z and z + 1,
// which lie side by side in a ring of plane accumulators in TMEM (NP planes; a
// window that wraps is issued in two parts).  An MMA costs the same issue time
// at N = 32 and 64 and little more at 96, so this halves the tensor time
// against one MMA per tap (9 x CIN/16 instead of 27 x CIN/16 per tile).  The
// order in which a plane's taps accumulate is that of the taps, (dz, dy, dx).
//
// Worker warps copy planes and run the epilogues (warps w, w + 4, .. read the
// same TMEM lanes, 32 (w % 4) .., and take 8 of the accumulator's columns each);
// one more warp issues the MMAs.  So while the tensor core runs input plane s,
// the workers start copying plane s + 2, finish the output plane that plane
// s - 1 completed and wait for plane s + 1: one block barrier per plane.
constexpr int kHX = 10, kHY = 18;
constexpr int kZWorkers = 256;             // copy threads of the weight gradient
constexpr int kZThreads = kZWorkers + 32;  // + the MMA warp
constexpr int kZIssuer = kZWorkers;        // the thread that issues the MMAs
constexpr int kEpiCols = 8;                // accumulator columns per worker thread
__host__ __device__ constexpr int conv_workers(int cout) { return kTileM * (cout / kEpiCols); }
__host__ __device__ constexpr int conv_threads(int cout) { return conv_workers(cout) + 32; }
constexpr int kSlots = 3;
__host__ __device__ constexpr int dhalo_slot_bytes(int cin) { return (cin / 8) * kHX * kHY * 16; }
__host__ __device__ constexpr int dhalo_bytes(int cin) { return kSlots * dhalo_slot_bytes(cin); }
// Accumulators in the TMEM ring: the three being summed and the one being read
// need 4; 8 where two blocks per SM leave the columns for it (fewer wraps).
__host__ __device__ constexpr int ring_planes(int cin, int cout) { return cin == 32 || cout == 16 ? 8 : 4; }
__host__ __device__ constexpr int ring_cols(int cin, int cout) { return ring_planes(cin, cout) * cout; }
__host__ __device__ inline bool dhalo_ok(int nx, int ny) { return nx % 8 == 0 && ny % 16 == 0; }

// Copies plane zz (-1 <= zz <= nz, periodic) of the column at (x0, y0) into
// its ring slot S (worker threads).
template <int CIN, int WORKERS>
__device__ __forceinline__ void dhalo_load_plane(const Grid3& g, const __nv_bfloat16* in, int x0,
                                                 int y0, int zz, unsigned char* S) {
    constexpr int N = (CIN / 8) * kHX * kHY;
    const int64_t zoff = (int64_t)wrapi(zz, g.nz) * g.ny;
    for (int i = threadIdx.x; i < N; i += WORKERS) {
        const int hx = i % kHX, hy = (i / kHX) % kHY, kg = i / (kHX * kHY);
        const int64_t cell = (zoff + wrapi(y0 - 1 + hy, g.ny)) * g.nx + wrapi(x0 - 1 + hx, g.nx);
        const uint4* src = reinterpret_cast<const uint4*>(in + cell * CIN) + kg;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(tc::smem_addr(S + i * 16)), "l"(src));
    }
}

// Epilogue of one tile: this thread's cell c (TMEM lane = threadIdx % 128)
// and its kEpiCols accumulator columns (bias: their biases).
template <int COUT, int MODE>
__device__ __forceinline__ void conv_epilogue(uint32_t tacc, int64_t c, int64_t V, const float (&bias)[kEpiCols],
                                              const __nv_bfloat16* __restrict__ pre_below,
                                              __nv_bfloat16* __restrict__ out_pre, __nv_bfloat16* __restrict__ out_bf,
                                              float* __restrict__ out_f) {
    constexpr int H = kEpiCols;
    static_assert(H == 8, "one 16-byte BF16 store per thread and cell");
    const int w = threadIdx.x >> 5, j0 = (threadIdx.x >> 7) * H;
    float acc[H];
    tc::tmem_ld8(tacc + ((uint32_t)(32 * (w & 3)) << 16) + (uint32_t)j0, acc);
    if constexpr (MODE == kFwdHidden) {
        __align__(16) __nv_bfloat16 pb[H], ab[H];
#pragma unroll
        for (int j = 0; j < H; ++j) {
            const float p = acc[j] + bias[j];
            pb[j] = __float2bfloat16(p);
            ab[j] = __float2bfloat16(gelu(p));
        }
        *reinterpret_cast<uint4*>(out_pre + c * COUT + j0) = *reinterpret_cast<const uint4*>(pb);
        *reinterpret_cast<uint4*>(out_bf + c * COUT + j0) = *reinterpret_cast<const uint4*>(ab);
    } else if constexpr (MODE == kFwdLast) {
        static_assert(MODE != kFwdLast || H == kOutChannels, "the columns from kOutChannels on are padding");
        if (j0 == 0) {
#pragma unroll
            for (int j = 0; j < H; ++j) out_f[j * V + c] = acc[j] + bias[j];
        }
    } else {
        __align__(16) __nv_bfloat16 pre[H], gb[H];
        *reinterpret_cast<uint4*>(pre) = *reinterpret_cast<const uint4*>(pre_below + c * COUT + j0);
#pragma unroll
        for (int j = 0; j < H; ++j) gb[j] = __float2bfloat16(acc[j] * gelu_grad(__bfloat162float(pre[j])));
        *reinterpret_cast<uint4*>(out_bf + c * COUT + j0) = *reinterpret_cast<const uint4*>(gb);
    }
}

// Block b marches column b % cols over planes [zc * (b / cols), + zc).
// Smem: B image, then the plane ring.
template <int CIN, int COUT, int MODE>
__global__ void __launch_bounds__(conv_threads(COUT)) conv_dhalo_kernel(Grid3 g, int zc, const __nv_bfloat16* in,
                                                               const uint4* __restrict__ bimg,
                                                               const float* __restrict__ bias,
                                                               const __nv_bfloat16* __restrict__ pre_below,
                                                               __nv_bfloat16* __restrict__ out_pre,
                                                               __nv_bfloat16* __restrict__ out_bf,
                                                               float* __restrict__ out_f, int* __restrict__ err,
                                                               uint32_t wait_limit) {
    constexpr int WORKERS = conv_workers(COUT), THREADS = conv_threads(COUT), ISSUER = WORKERS;
    constexpr int KS = CIN / 16;
    constexpr int BBYTES = bimg_bytes(CIN, COUT);
    constexpr int SLOT = dhalo_slot_bytes(CIN);
    constexpr int NP = ring_planes(CIN, COUT), TCOLS = ring_cols(CIN, COUT);
    constexpr uint32_t KG = kHX * kHY;  // 16-byte units between 8-channel groups
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ uint64_t bar[2];
    __shared__ uint32_t tslot;
    unsigned char* Bs = sm;
    unsigned char* Hs = sm + BBYTES;
    const int t = threadIdx.x;
    const int bx = g.nx / 8, cols = bx * (g.ny / 16);
    const int col = (int)(blockIdx.x % (unsigned)cols);
    const int x0 = (col % bx) * 8, y0 = (col / bx) * 16;
    const int za = (int)(blockIdx.x / (unsigned)cols) * zc, len = min(zc, g.nz - za);
    const int last = len + 1;  // steps 0 .. last: input planes za - 1 .. za + len
    const bool worker = t < WORKERS;
    // What no kernel still running writes (weights, biases) comes before
    // pdl_begin(), the input planes after it.
    for (int i = t; i < BBYTES / 16; i += THREADS)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(tc::smem_addr(Bs + i * 16)), "l"(bimg + i));
    if (t == 0) {
        tc::mbar_init(&bar[0], 1);
        tc::mbar_init(&bar[1], 1);
        tc::mbar_fence_init();
    }
    if (t < 32) tc::tmem_alloc(&tslot, TCOLS);
    float bias_h[kEpiCols];  // the biases of this worker's columns
#pragma unroll
    for (int j = 0; j < kEpiCols; ++j)
        bias_h[j] = (MODE != kBwdData && worker) ? bias[(t >> 7) * kEpiCols + j] : 0.0f;
    pdl_begin();
    if (worker) {
        dhalo_load_plane<CIN, WORKERS>(g, in, x0, y0, za - 1, Hs);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        dhalo_load_plane<CIN, WORKERS>(g, in, x0, y0, za, Hs + SLOT);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // weights and plane za - 1 in; za may be in flight
    } else {
        asm volatile("cp.async.wait_all;\n" ::: "memory");
    }
    tc::fence_smem_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tslot;
    const uint32_t h0 = tc::smem_addr(Hs), b0 = tc::smem_addr(Bs);
    // a worker's cell in a tile of plane z: M row t % 128
    const int64_t nxy = (int64_t)g.nx * g.ny;
    const int64_t cxy = (int64_t)(y0 + (t & 127) / 8) * g.nx + x0 + (t & 7);
    bool ok = true;
    int n = 0;  // steps issued
    for (int s = 0; s <= last && ok; ++s) {
        if (t == ISSUER) {
            // Input plane r (relative to za) feeds the output planes lo .. hi of
            // r - 1 .. r + 1; the last of them, r + 1, starts with this plane.
            const int r = s - 1, lo = max(r - 1, 0), hi = min(r + 1, len - 1);
            const bool fresh = r + 1 <= len - 1;
            // the window's accumulators: n0 planes at slot lo % NP, the rest (if
            // it wraps) from slot 0 on
            const int n0 = min(hi - lo + 1, NP - lo % NP), n1 = hi - lo + 1 - n0;
            const uint32_t d0 = tmem + (uint32_t)(lo % NP) * COUT;
            const uint32_t i0 = tc::idesc_bf16(kTileM, COUT, 0, 0) + (uint32_t)((n0 - 1) * (COUT / 8)) * (1u << 17);
            const uint32_t i1 = tc::idesc_bf16(kTileM, COUT, 0, 0) + (uint32_t)((n1 - 1) * (COUT / 8)) * (1u << 17);
            // descriptors: the start address is the low field (16-byte units,
            // smem < 256 KB so no carry), offsets add directly
            const uint64_t da0 = tc::smem_desc(h0 + (s % kSlots) * SLOT, KG * 16, kHX * 16);
            const uint64_t db0 = tc::smem_desc(b0 + (uint32_t)(lo - (r - 1)) * COUT * 32, 128, 256);
#pragma unroll
            for (int yx = 0; yx < 9; ++yx) {
#pragma unroll
                for (int kb = 0; kb < KS; ++kb) {
                    const uint64_t da = da0 + (uint32_t)(2 * kb * KG + (yx / 3) * kHX + yx % 3);
                    const uint64_t db = db0 + (uint32_t)((yx * KS + kb) * 3 * COUT * 32 / 16);
                    if (yx == 0 && kb == 0 && fresh) {
                        // one plane at a time: plane r + 1 overwrites its slot
                        for (int o = lo; o <= hi; ++o)
                            tc::mma_bf16(tmem + (uint32_t)(o % NP) * COUT, da, db + (uint32_t)((o - lo) * COUT * 32 / 16),
                                         tc::idesc_bf16(kTileM, COUT, 0, 0), o <= r ? 1u : 0u);
                    } else {
                        tc::mma_bf16(d0, da, db, i0, 1u);
                        if (n1 > 0) tc::mma_bf16(tmem, da, db + (uint32_t)(n0 * COUT * 32 / 16), i1, 1u);
                    }
                }
            }
            tc::mma_commit(&bar[s & 1]);
        }
        n = s + 1;
        bool lost = false;
        if (worker) {
            // step s - 1 done: its plane's slot takes plane s + 2, and output
            // plane s - 3 is final
            if (s > 0) lost = !tc::mbar_wait(&bar[(s - 1) & 1], ((s - 1) >> 1) & 1, err, wait_limit);
            if (!lost) {
                tc::fence_after_sync();
                if (s + 2 <= last)
                    dhalo_load_plane<CIN, WORKERS>(g, in, x0, y0, za + s + 1, Hs + ((s + 2) % kSlots) * SLOT);
                asm volatile("cp.async.commit_group;\n" ::: "memory");
                if (s >= 3)
                    conv_epilogue<COUT, MODE>(tmem + (uint32_t)((s - 3) % NP) * COUT, (int64_t)(za + s - 3) * nxy + cxy,
                                              g.V, bias_h, pre_below, out_pre, out_bf, out_f);
            }
            // plane s + 1 in; s + 2 may stay in flight
            if (lost) asm volatile("cp.async.wait_all;\n" ::: "memory");
            else asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            tc::fence_smem_async();
        }
        tc::fence_before_sync();
        if (__syncthreads_or(lost)) {  // plane s + 1 visible; accumulator s - 3 read
            ok = false;
            break;
        }
        tc::fence_after_sync();
    }
    if (ok) {
        bool lost = false;
        if (worker) lost = !tc::mbar_wait(&bar[last & 1], (last >> 1) & 1, err, wait_limit);
        if (!__syncthreads_or(lost) && worker) {
            tc::fence_after_sync();
            conv_epilogue<COUT, MODE>(tmem + (uint32_t)((len - 1) % NP) * COUT, (int64_t)(za + len - 1) * nxy + cxy, g.V,
                                      bias_h, pre_below, out_pre, out_bf, out_f);
        }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");  // no copy outlives the block
    if (t == 0) {  // drain: the newest commit on each barrier
        for (int k = 1; k <= 2; ++k)
            if (n >= k) tc::mbar_wait(&bar[(n - k) & 1], ((n - k) >> 1) & 1, err);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (t < 32) tc::tmem_dealloc(tmem, TCOLS);
}

// Weight gradient dW[tap][ci][co] = sum_c act[c + off(tap)][ci] * grad[c][co]
// over this CTA's cell range, as partials[cta][tap][ci][co] (FP32).
// M rows = (tap-in-group j, ci), TPG = 128/CIN taps per group, G groups;
// K = cells, 32 per stage (2 k-steps); operands MN-major.
template <int CIN, int COUT>
struct WGradShape {
    static constexpr int TPG = kTileM / CIN;
    static constexpr int G = (27 + TPG - 1) / TPG;
    static constexpr int COLS = G * COUT;
    static constexpr int TCOLS = COLS <= 32 ? 32 : (COLS <= 64 ? 64 : (COLS <= 128 ? 128 : 256));
    static constexpr int KC = 32;                                  // cells per stage
    static constexpr int ABLK = 4096;                              // 128 x 16 BF16
    static constexpr int BBLK = COUT * 32;                         // COUT x 16 BF16
    static constexpr int STAGE = G * 2 * ABLK + 2 * BBLK;
    static constexpr int SMEM = 2 * STAGE;
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(kThreads) wgrad_kernel(Grid3 g, const __nv_bfloat16* __restrict__ act,
                                                         const __nv_bfloat16* __restrict__ grad,
                                                         float* __restrict__ partials, int* __restrict__ err,
        uint32_t wait_limit) {
    using WS = WGradShape<CIN, COUT>;
    constexpr int TPG = WS::TPG, G = WS::G, KC = WS::KC;
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ uint64_t bar[2];
    __shared__ uint32_t tslot;
    const int t = threadIdx.x;
    if (t == 0) {
        tc::mbar_init(&bar[0], 1);
        tc::mbar_init(&bar[1], 1);
        tc::mbar_fence_init();
    }
    if (t < 32) tc::tmem_alloc(&tslot, WS::TCOLS);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tslot;
    const uint32_t idesc = tc::idesc_bf16(kTileM, COUT, 1, 1);
    const uint32_t s0 = tc::smem_addr(sm);
    uint32_t uses[2] = {0, 0};
    bool ok = true;

    const int64_t nchunks = (g.V + KC - 1) / KC;
    const int64_t ch0 = nchunks * blockIdx.x / gridDim.x, ch1 = nchunks * (blockIdx.x + 1) / gridDim.x;
    bool first = true;
    for (int64_t ch = ch0; ch < ch1; ++ch) {
        const int s = (int)((ch - ch0) & 1);
        bool lost = uses[s] > 0 && !tc::mbar_wait(&bar[s], (uses[s] - 1) & 1, err, wait_limit);
        if (__syncthreads_or(lost)) {
            ok = false;
            break;
        }
        unsigned char* st = sm + s * WS::STAGE;
        // A: item = (slot = tap slot of 28 or 32, q = ci chunk of 8, k = cell of KC)
        constexpr int NA = G * TPG * (CIN / 8) * KC;
        for (int i = t; i < NA; i += kThreads) {
            const int q = i % (CIN / 8);
            const int k = (i / (CIN / 8)) % KC;
            const int slot = i / ((CIN / 8) * KC);
            const int gi = slot / TPG, j = slot % TPG;
            const int64_t c = ch * KC + k;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (slot < 27 && c < g.V) {
                const int x = (int)(c % g.nx), y = (int)((c / g.nx) % g.ny), z = (int)(c / ((int64_t)g.nx * g.ny));
                v = reinterpret_cast<const uint4*>(act + neighbour(g, x, y, z, slot) * CIN)[q];
            }
            const int m = j * CIN + q * 8;
            const int kk = k % 16;
            *reinterpret_cast<uint4*>(st + (gi * 2 + k / 16) * WS::ABLK + (m / 8) * 128 + (kk / 8) * 2048 +
                                      (kk % 8) * 16) = v;
        }
        // B: item = (q = co chunk of 8, k)
        unsigned char* bst = st + G * 2 * WS::ABLK;
        for (int i = t; i < (COUT / 8) * KC; i += kThreads) {
            const int q = i % (COUT / 8), k = i / (COUT / 8);
            const int64_t c = ch * KC + k;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (c < g.V) v = reinterpret_cast<const uint4*>(grad + c * COUT)[q];
            const int kk = k % 16;
            *reinterpret_cast<uint4*>(bst + (k / 16) * WS::BBLK + q * 128 + (kk / 8) * (COUT / 8) * 128 +
                                      (kk % 8) * 16) = v;
        }
        tc::fence_smem_async();
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
        if (t == 0) {
            const uint32_t sa = s0 + s * WS::STAGE;
#pragma unroll 1
            for (int gi = 0; gi < G; ++gi) {
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) {
                    const uint64_t da = tc::smem_desc(sa + (gi * 2 + ks) * WS::ABLK, 2048, 128);
                    const uint64_t db = tc::smem_desc(sa + G * 2 * WS::ABLK + ks * WS::BBLK, (COUT / 8) * 128, 128);
                    tc::mma_bf16(tmem + gi * COUT, da, db, idesc, (first && ks == 0) ? 0u : 1u);
                }
            }
            tc::mma_commit(&bar[s]);
        }
        first = false;
        ++uses[s];
    }
    if (ok && uses[0] + uses[1] > 0) {
        const int last = (int)(((ch1 - ch0) - 1) & 1);
        const bool lost = !tc::mbar_wait(&bar[last], (uses[last] - 1) & 1, err, wait_limit);
        ok = !__syncthreads_or(lost);
    }
    tc::fence_after_sync();
    if (ok) {
        const int w = t >> 5;
        const int j = t / CIN, ci = t % CIN;
        float* dst = partials + (int64_t)blockIdx.x * 27 * CIN * COUT;
        for (int gi = 0; gi < G; ++gi) {
            float v[COUT];
            if (first) {
#pragma unroll
                for (int co = 0; co < COUT; ++co) v[co] = 0.0f;  // no cells: zero partial
            } else {
#pragma unroll
                for (int c0 = 0; c0 < COUT; c0 += 16)
                    tc::tmem_ld16(tmem + ((uint32_t)(32 * w) << 16) + (uint32_t)(gi * COUT + c0), v + c0);
            }
            const int tap = gi * TPG + j;
            if (tap < 27) {
#pragma unroll
                for (int co = 0; co < COUT; ++co) dst[((int64_t)tap * CIN + ci) * COUT + co] = v[co];
            }
        }
    }
    if (t == 0) {
        for (int s = 0; s < 2; ++s)
            if (uses[s] > 0) tc::mbar_wait(&bar[s], (uses[s] - 1) & 1, err);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (t < 32) tc::tmem_dealloc(tmem, WS::TCOLS);
}

// Weight gradient on 8 x 16 x 1 tiles (nx % 8 == 0, ny % 16 == 0), marching z.
//
// dW[tap][ci][co] is a GEMM with M = (tap, ci), N = co and K = cells.  The
// tensor core reads both operands where cp.async put them: an MN-major core
// matrix holds 8 channels of 8 consecutive cells, 16 bytes per cell, which is
// what 8 x-cells of a channel-last field are.  A staged plane holds three
// copies of the column's 18 rows, shifted by dx = -1, 0, 1, each 8 cells wide
// and one block per 8-channel group:
//   unit(slot, g, hy, x) at slot*SLOT + (g*18 + hy)*8 + x,  g = (dx+1)*CIN/8 + kg,
// so 16 consecutive groups at one stride are the M = 128 rows of an operand:
// the 3 CIN rows of the three dx taps, and groups of the next slot whose rows
// are not read back.  dy moves the start by one row (128 bytes), dz picks the
// slot, and the K groups (y rows) are 128 bytes apart.  A tile is 9 (dy, dz) x 8
// K-steps of MMAs and costs one new plane and one gradient tile; nothing is
// copied inside shared memory.  (Assembling a 32 KB operand per 4 taps in shared
// memory instead took 179 us per 32 -> 32 layer at 64^3, and the bias gradient
// 25 us in kernels of its own.)
//
// One block per SM takes an equal share of the column-major sequence of tiles.
// Warps 0-7 copy (two planes ahead, ring of 5 planes and 3 gradient tiles),
// warp 8 issues the MMAs; one block barrier per tile.  The nine accumulators
// (COUT columns each) stay in TMEM for half of the share: the tensor core's FP32
// sums drift with their length, and the halves, added in FP32, are as long as
// the sums of two blocks per SM.  The bias gradient, which needs no product, is
// summed by the copying warps from the staged tiles in FP32.  Error against 64
// bits at 80^3, of the sum of the terms' magnitudes, weights / biases: 1.8e-6 /
// 7e-8; whole shares with the biases as a row of the product 5.0e-6 / 4.4e-7, in
// 57 us for the 64 us a 32 -> 32 layer takes at 64^3.
constexpr int kWRing = 5, kWGrads = 3;
template <int CIN, int COUT>
struct WGradMarch {
    static constexpr int KGN = CIN / 8;
    static constexpr int GROUP = kHY * 8 * 16;             // bytes of one channel group
    static constexpr int SLOTG = 3 * KGN;                  // groups per plane
    static constexpr int SLOT = SLOTG * GROUP;
    static constexpr int PAD = (16 - SLOTG) * GROUP;       // the last slot's operand ends here
    static constexpr int GB = (COUT / 8) * 2048;           // output-gradient tile
    static constexpr int SMEM = kWRing * SLOT + PAD + kWGrads * GB;
    static constexpr int TCOLS = 9 * COUT <= 256 ? 256 : 512;
    static constexpr int NOUT = 27 * CIN * COUT + COUT;    // weights, then biases
    static_assert(SLOTG <= 16, "a plane's groups lie inside the 128 operand rows");
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(kZThreads) wgrad_march_kernel(Grid3 g, const __nv_bfloat16* act,
                                                                const __nv_bfloat16* grad,
                                                                float* __restrict__ partials, int* __restrict__ err,
                                                                uint32_t wait_limit) {
    using WM = WGradMarch<CIN, COUT>;
    constexpr int KGN = WM::KGN, SLOT = WM::SLOT;
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ uint64_t bar[2];
    __shared__ uint32_t tslot;
    unsigned char* Gs = sm + kWRing * SLOT + WM::PAD;
    const int t = threadIdx.x;
    if (t == 0) {
        tc::mbar_init(&bar[0], 1);
        tc::mbar_init(&bar[1], 1);
        tc::mbar_fence_init();
    }
    if (t < 32) tc::tmem_alloc(&tslot, WM::TCOLS);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    pdl_begin();
    const uint32_t tmem = tslot;
    const uint32_t idesc = tc::idesc_bf16(kTileM, COUT, 1, 1);
    const uint32_t s0 = tc::smem_addr(sm), g0 = tc::smem_addr(Gs);
    const bool worker = t < kZWorkers;
    const int bx = g.nx / 8;
    const int64_t ntiles = (int64_t)bx * (g.ny / 16) * g.nz;
    const int64_t tile0 = ntiles * blockIdx.x / gridDim.x;  // gridDim.x <= ntiles: no share is empty
    const int64_t tile1 = ntiles * (blockIdx.x + 1) / gridDim.x;
    const int64_t mid = tile0 + (tile1 - tile0 + 1) / 2;
    int64_t tile = tile0;
    int n = 0;  // tiles issued by this block
    bool ok = true;
    float* const dst = partials + (int64_t)blockIdx.x * WM::NOUT;
    // The accumulators into this block's partials (MarchOrder), or added to them
    // (workers).  Warps w and w + 4 read the same lanes and take alternate
    // accumulators.
    auto flush = [&](bool add) {
        const int w = t >> 5, m = t & 127;
        for (int gi = w >> 2; gi < 9; gi += 2) {
            float v[COUT];
#pragma unroll
            for (int c0 = 0; c0 < COUT; c0 += 16)
                tc::tmem_ld16(tmem + ((uint32_t)(32 * (w & 3)) << 16) + (uint32_t)(gi * COUT + c0), v + c0);
            if (m < 3 * CIN) {
                float4* o = reinterpret_cast<float4*>(dst) + gi * (COUT / 4) * 3 * CIN + m;
#pragma unroll
                for (int q = 0; q < COUT / 4; ++q) {
                    float4 s = add ? o[q * 3 * CIN] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    s.x += v[4 * q];
                    s.y += v[4 * q + 1];
                    s.z += v[4 * q + 2];
                    s.w += v[4 * q + 3];
                    o[q * 3 * CIN] = s;
                }
            }
            __syncwarp();  // the next load is a whole warp's
        }
    };
    // Bias gradient: warp w sums channel group w % NG of a gradient tile
    constexpr int NG = COUT / 8, BC = (kZWorkers / 32) / NG;  // groups; warps per group
    float bsum[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    while (tile < tile1 && ok) {
        // one column segment: planes [za, za + len)
        const int64_t col = tile / g.nz;
        const int za = (int)(tile - col * g.nz);
        const int len = (int)min((int64_t)(g.nz - za), (tile < mid ? mid : tile1) - tile);
        const bool fresh = tile == tile0 || tile == mid;  // starts new sums
        const int x0 = (int)(col % bx) * 8, y0 = (int)(col / bx) * 16;
        // plane za + r (-1 <= r <= len) into slot (r + 1) % ring, gradient tile
        // za + r into slot r % 3
        auto load_plane = [&](int r) {
            unsigned char* S = sm + ((r + 1) % kWRing) * SLOT;
            const int64_t zoff = (int64_t)wrapi(za + r, g.nz) * g.ny;
            for (int i = t; i < 3 * KGN * kHY * 8; i += kZWorkers) {
                const int x = i % 8, hy = (i / 8) % kHY, gr = i / (8 * kHY);
                const int dx = gr / KGN - 1, kg = gr % KGN;
                const int64_t cell = (zoff + wrapi(y0 - 1 + hy, g.ny)) * g.nx + wrapi(x0 + x + dx, g.nx);
                const uint4* src = reinterpret_cast<const uint4*>(act + cell * CIN) + kg;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(tc::smem_addr(S + i * 16)), "l"(src));
            }
        };
        auto load_grad = [&](int r) {
            unsigned char* D = Gs + (r % kWGrads) * WM::GB;
            for (int i = t; i < (COUT / 8) * 128; i += kZWorkers) {
                const int k = i % 128, q = i / 128;
                const int64_t cell = ((int64_t)(za + r) * g.ny + y0 + k / 8) * g.nx + x0 + k % 8;
                const uint4* src = reinterpret_cast<const uint4*>(grad + cell * COUT) + q;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(tc::smem_addr(D + i * 16)), "l"(src));
            }
        };
        bool lost = false;
        if (worker) {
            // the previous segment's MMAs read the slots refilled here
            if (n > 0) lost = !tc::mbar_wait(&bar[(n - 1) & 1], ((n - 1) >> 1) & 1, err, wait_limit);
            if (!lost) {
                for (int r = -1; r <= 1; ++r) load_plane(r);
                load_grad(0);
                asm volatile("cp.async.commit_group;\n" ::: "memory");
                if (len > 1) {
                    load_plane(2);
                    load_grad(1);
                }
                asm volatile("cp.async.commit_group;\n" ::: "memory");
                if (fresh && n > 0) {  // the first half's sums are final
                    tc::fence_after_sync();
                    flush(false);
                }
                asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            }
            tc::fence_smem_async();
        }
        tc::fence_before_sync();
        if (__syncthreads_or(lost)) {
            ok = false;
            break;
        }
        tc::fence_after_sync();
        for (int i = 0; i < len; ++i, ++n) {
            if (t == kZIssuer) {
                const uint64_t db0 = tc::smem_desc(g0 + (i % kWGrads) * WM::GB, 128, 2048);
#pragma unroll
                for (int gi = 0; gi < 9; ++gi) {
                    const int dy = gi % 3 - 1, dz = gi / 3 - 1;
                    const uint64_t da0 =
                        tc::smem_desc(s0 + ((i + dz + 1) % kWRing) * SLOT + (1 + dy) * 128, 128, WM::GROUP);
#pragma unroll
                    for (int ks = 0; ks < 8; ++ks)
                        tc::mma_bf16(tmem + gi * COUT, da0 + (uint32_t)(ks * 256 / 16), db0 + (uint32_t)(ks * 256 / 16),
                                     idesc, (!fresh || i > 0 || ks > 0) ? 1u : 0u);
                }
                tc::mma_commit(&bar[n & 1]);
            }
            if (worker) {
                // this tile's gradient was complete at the last barrier and keeps its
                // slot until the next one
                const unsigned char* D = Gs + (i % kWGrads) * WM::GB + ((t >> 5) % NG) * 2048;
                for (int k = (t >> 5) / NG * 32 + (t & 31); k < kTileM; k += 32 * BC) {
                    const uint4 u = *reinterpret_cast<const uint4*>(D + k * 16);
                    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 f = __bfloat1622float2(h[j]);
                        bsum[2 * j] += f.x;
                        bsum[2 * j + 1] += f.y;
                    }
                }
                // tile n - 1 done: plane i - 2 (its slot takes plane i + 3) and
                // the gradient of tile i - 1 are no longer read
                if (n > 0) lost = !tc::mbar_wait(&bar[(n - 1) & 1], ((n - 1) >> 1) & 1, err, wait_limit);
                if (!lost) {
                    if (i + 3 <= len) load_plane(i + 3);
                    if (i + 2 < len) load_grad(i + 2);
                    asm volatile("cp.async.commit_group;\n" ::: "memory");
                    asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // plane i + 2, gradient i + 1
                } else {
                    asm volatile("cp.async.wait_all;\n" ::: "memory");
                }
                tc::fence_smem_async();
            }
            tc::fence_before_sync();
            if (__syncthreads_or(lost)) {
                ok = false;
                ++n;
                break;
            }
            tc::fence_after_sync();
        }
        tile += len;
    }
    if (ok && n > 0) {
        const bool lost = !tc::mbar_wait(&bar[(n - 1) & 1], ((n - 1) >> 1) & 1, err, wait_limit);
        ok = !__syncthreads_or(lost);
    }
    tc::fence_after_sync();
    __shared__ float bsh[kZWorkers / 32][8];
    if (ok && worker) {
        flush(mid < tile1);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float v = bsum[j];
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if ((t & 31) == 0) bsh[t >> 5][j] = v;
        }
    }
    __syncthreads();
    if (ok && t < COUT) {
        float v = 0.0f;
        for (int w = t / 8; w < kZWorkers / 32; w += NG) v += bsh[w][t % 8];
        dst[27 * CIN * COUT + t] = v;
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");  // no copy outlives the block
    if (t == 0) {  // drain: the newest commit on each barrier
        for (int k = 1; k <= 2; ++k)
            if (n >= k) tc::mbar_wait(&bar[(n - k) & 1], ((n - k) >> 1) & 1, err);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (t < 32) tc::tmem_dealloc(tmem, WM::TCOLS);
}

// Order of a block's partials: the gradient's own, [tap][ci][co] and then the
// biases, or wgrad_march_kernel's, where the lanes of an accumulator store
// neighbouring float4: accumulator (dy, dz), 4 columns, lane (dx, ci), column.
struct GradOrder {
    __device__ __forceinline__ int operator()(int j) const { return j; }
};
template <int CIN, int COUT>
struct MarchOrder {
    __device__ __forceinline__ int operator()(int j) const {
        if (j >= 27 * CIN * COUT) return j;
        const int e = j % 4, m = j / 4 % (3 * CIN), k = j / (12 * CIN), q = k % (COUT / 4), gi = k / (COUT / 4);
        return ((gi * 3 + m / CIN) * CIN + m % CIN) * COUT + 4 * q + e;
    }
};

// out[order(j)] = sum over p < P of partials[p * n + j] in a fixed order: a block
// takes 32 consecutive j; its warp s sums the partials p = s, s + 8, ... in
// increasing p, then the 8 slice sums are added in increasing s.  (One
// thread per j summing all P serially left most SMs idle.)  Launch with
// kFoldThreads threads and ceil(n / 32) blocks.
constexpr int kFoldThreads = 256;
template <class Order>
__global__ void __launch_bounds__(kFoldThreads) sum_partials_kernel(const float* partials, int P, int n,
                                                                     float* __restrict__ out) {
    __shared__ float slice[kFoldThreads / 32][32];
    const int lane = threadIdx.x & 31, s = threadIdx.x >> 5;
    const int j = blockIdx.x * 32 + lane;
    pdl_begin();
    float acc = 0.0f;
    if (j < n)
        for (int p = s; p < P; p += kFoldThreads / 32) acc += partials[(int64_t)p * n + j];
    slice[s][lane] = acc;
    __syncthreads();
    if (s == 0 && j < n) {
        float t = slice[0][lane];
#pragma unroll
        for (int k = 1; k < kFoldThreads / 32; ++k) t += slice[k][lane];
        out[Order()(j)] = t;
    }
}

// Bias gradient partials: per block, sum over its cells of grad[c][co].
template <int C>
__global__ void bias_grad_kernel(const __nv_bfloat16* __restrict__ grad, int64_t V, float* __restrict__ partials) {
    __shared__ float sh[kThreads / 32][C];
    float acc[C];
#pragma unroll
    for (int j = 0; j < C; ++j) acc[j] = 0.0f;
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < V; c += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
        for (int j = 0; j < C; ++j) acc[j] += __bfloat162float(grad[c * C + j]);
    }
#pragma unroll
    for (int j = 0; j < C; ++j) {
        float v = acc[j];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5][j] = v;
    }
    __syncthreads();
    if (threadIdx.x < C) {
        float v = 0.0f;
        for (int w = 0; w < kThreads / 32; ++w) v += sh[w][threadIdx.x];
        partials[(int64_t)blockIdx.x * C + threadIdx.x] = v;
    }
}

// Fwd and backward-data B images of one layer from the FP32 master weights
// W[27][CIN][COUT] (padding rows/columns are zero in the master copy).
template <int CIN, int COUT>
__global__ void pack_kernel(const float* __restrict__ W, __nv_bfloat16* __restrict__ fwd,
                            __nv_bfloat16* __restrict__ bwd) {
    const int n = 27 * CIN * COUT;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int co = i % COUT, ci = (i / COUT) % CIN, tap = i / (CIN * COUT);
        const __nv_bfloat16 v = __float2bfloat16(W[i]);
        {  // forward: B[n = co][k = ci] of k-step (tap, ci/16)
            const int k = ci % 16;
            fwd[(bimg_off(CIN, COUT, tap % 9, ci / 16, tap / 9 - 1) + tc::kmajor_off(co, k, 128, 256)) / 2] = v;
        }
        if (bwd) {  // backward data: tap' = 26 - tap, B[n = ci][k = co]
            const int tp = 26 - tap, k = co % 16;
            bwd[(bimg_off(COUT, CIN, tp % 9, co / 16, tp / 9 - 1) + tc::kmajor_off(ci, k, 128, 256)) / 2] = v;
        }
    }
}

// Adam on the flat FP32 parameter vector.
__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ grad, float* __restrict__ m,
                            float* __restrict__ v, const float* __restrict__ mask, int n, float lr, float b1,
                            float b2, float eps, float bc1, float bc2) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float gi = grad[i] * mask[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= mask[i] * lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    }
}

// Standard normal variate from a counter (splitmix64 of key and index,
// Box-Muller), for training-input noise.
__device__ __forceinline__ float hash_normal(uint64_t key, uint64_t i) {
    auto mix = [](uint64_t z) {
        z += 0x9e3779b97f4a7c15ull;
        z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
        z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
        return z ^ (z >> 31);
    };
    const uint64_t h = mix(key ^ mix(i));
    const float u1 = ((float)(h >> 40) + 0.5f) * 0x1.0p-24f, u2 = (float)((h >> 16) & 0xFFFFFF) * 0x1.0p-24f;
    return sqrtf(-2.0f * logf(u1)) * cospif(2.0f * u2);
}

// Network input from 9 FP32 channel blocks (rho, u, Q; [9][V]):
// act0[c][j] = (x_j - shift_j) * inv_scale_j (+ noise_std N(0,1) when
// training with input noise) for j < 9, 0 for j in 9..15.
__global__ void features_kernel(const float* rho, const float* u3,
                                const float* q5, int64_t V, const float* __restrict__ shift,
                                const float* __restrict__ inv_scale, __nv_bfloat16* __restrict__ act0,
                                float noise_std, uint64_t noise_key) {
    pdl_begin();
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < V; c += (int64_t)gridDim.x * blockDim.x) {
        __align__(16) __nv_bfloat16 v[16];
        float x[9];
        x[0] = rho[c];
#pragma unroll
        for (int k = 0; k < 3; ++k) x[1 + k] = u3[k * V + c];
#pragma unroll
        for (int k = 0; k < 5; ++k) x[4 + k] = q5[k * V + c];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            float f = 0.0f;
            if (j < 9) {
                f = (x[j] - shift[j]) * inv_scale[j];
                if (noise_std > 0.0f) f += noise_std * hash_normal(noise_key, (uint64_t)c * 16 + j);
            }
            v[j] = __float2bfloat16(f);
        }
        reinterpret_cast<uint4*>(act0 + c * 16)[0] = reinterpret_cast<const uint4*>(v)[0];
        reinterpret_cast<uint4*>(act0 + c * 16)[1] = reinterpret_cast<const uint4*>(v)[1];
    }
}

// Mean-squared error of the 8 outputs against the raw targets [8][V]
// normalised by inv_scale, its gradient gout[c][16] (BF16, channels 8..15
// zero) and per-block partial sums of the squared error.
__global__ void __launch_bounds__(kThreads) loss_kernel(const float* out, const float* tgt,
                                                        const float* __restrict__ inv_scale, int64_t V,
                                                        __nv_bfloat16* __restrict__ gout,
                                                        double* __restrict__ partials) {
    __shared__ double sh[kThreads / 32];
    double acc = 0.0;
    const float gscale = 2.0f / (8.0f * (float)V);
    pdl_begin();
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < V; c += (int64_t)gridDim.x * blockDim.x) {
        __align__(16) __nv_bfloat16 gv[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            float gj = 0.0f;
            if (j < 8) {
                const float d = out[j * V + c] - tgt[j * V + c] * inv_scale[j];
                acc += (double)d * d;
                gj = gscale * d;
            }
            gv[j] = __float2bfloat16(gj);
        }
        reinterpret_cast<uint4*>(gout + c * 16)[0] = reinterpret_cast<const uint4*>(gv)[0];
        reinterpret_cast<uint4*>(gout + c * 16)[1] = reinterpret_cast<const uint4*>(gv)[1];
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double v = 0.0;
        for (int w = 0; w < kThreads / 32; ++w) v += sh[w];
        partials[blockIdx.x] = v;
    }
}

// Correction of a coarse state after its step: Q_k += gain out[k][c] s_k
// (k < 5), u_d += gain out[5+d][c] s_{5+d}.
__global__ void apply_kernel(const float* out, const float* __restrict__ out_scale, int64_t V,
                             float gain, float* __restrict__ u3, float* __restrict__ q5) {
    pdl_begin();
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < V; c += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
        for (int k = 0; k < 5; ++k) q5[k * V + c] += gain * out[k * V + c] * out_scale[k];
#pragma unroll
        for (int d = 0; d < 3; ++d) u3[d * V + c] += gain * out[(5 + d) * V + c] * out_scale[5 + d];
    }
}

// Box filter of a fine state (factor f per axis) onto the coarse grid:
// rho_c = <rho>, u_c = <rho u> / rho_c, Q_c = <Q>; out [9][Vc].
__global__ void filter_kernel(const float* __restrict__ rho, const float* __restrict__ u3,
                              const float* __restrict__ q5, int nx, int ny, int nz, int f,
                              float* __restrict__ out) {
    const int cx = nx / f, cy = ny / f, cz = nz / f;
    const int64_t Vc = (int64_t)cx * cy * cz, V = (int64_t)nx * ny * nz;
    const double inv = 1.0 / ((double)f * f * f);
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < Vc; c += (int64_t)gridDim.x * blockDim.x) {
        const int X = (int)(c % cx), Y = (int)((c / cx) % cy), Z = (int)(c / ((int64_t)cx * cy));
        double r = 0, m[3] = {0, 0, 0}, q[5] = {0, 0, 0, 0, 0};
        for (int dz = 0; dz < f; ++dz)
            for (int dy = 0; dy < f; ++dy)
                for (int dx = 0; dx < f; ++dx) {
                    const int64_t i = ((int64_t)(Z * f + dz) * ny + (Y * f + dy)) * nx + (X * f + dx);
                    const double ri = rho[i];
                    r += ri;
#pragma unroll
                    for (int d = 0; d < 3; ++d) m[d] += ri * u3[d * V + i];
#pragma unroll
                    for (int k = 0; k < 5; ++k) q[k] += q5[k * V + i];
                }
        out[c] = (float)(r * inv);
#pragma unroll
        for (int d = 0; d < 3; ++d) out[(1 + d) * Vc + c] = (float)(m[d] / r);
#pragma unroll
        for (int k = 0; k < 5; ++k) out[(4 + k) * Vc + c] = (float)(q[k] * inv);
    }
}

// Per-block sums and sums of squares of nc channel blocks [nc][V] (or a
// difference a - b when b is given): partials[(blk * nc + j) * 2 + {0,1}].
__global__ void __launch_bounds__(kThreads) moments_kernel(const float* __restrict__ a, const float* __restrict__ b,
                                                           int nc, int64_t V, double* __restrict__ partials) {
    __shared__ double sh[2][kThreads / 32];
    for (int j = 0; j < nc; ++j) {
        double s1 = 0.0, s2 = 0.0;
        for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < V;
             c += (int64_t)gridDim.x * blockDim.x) {
            const double x = (double)a[j * V + c] - (b ? (double)b[j * V + c] : 0.0);
            s1 += x;
            s2 += x * x;
        }
        for (int o = 16; o > 0; o >>= 1) {
            s1 += __shfl_xor_sync(0xffffffffu, s1, o);
            s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        }
        if ((threadIdx.x & 31) == 0) {
            sh[0][threadIdx.x >> 5] = s1;
            sh[1][threadIdx.x >> 5] = s2;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double v1 = 0.0, v2 = 0.0;
            for (int w = 0; w < kThreads / 32; ++w) {
                v1 += sh[0][w];
                v2 += sh[1][w];
            }
            partials[((int64_t)blockIdx.x * nc + j) * 2] = v1;
            partials[((int64_t)blockIdx.x * nc + j) * 2 + 1] = v2;
        }
        __syncthreads();
    }
}

// Raw training target [8][V]: next - pred, Q components then u.
__global__ void target_kernel(const float* __restrict__ next9, const float* __restrict__ pu3,
                              const float* __restrict__ pq5, int64_t V, float* __restrict__ tgt) {
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < V; c += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
        for (int k = 0; k < 5; ++k) tgt[k * V + c] = next9[(4 + k) * V + c] - pq5[k * V + c];
#pragma unroll
        for (int d = 0; d < 3; ++d) tgt[(5 + d) * V + c] = next9[(1 + d) * V + c] - pu3[d * V + c];
    }
}

}  // namespace cl
}  // namespace lbman
