// api.cu -- the C ABI of include/lbman3d.h: device memory, launch sequencing
// and error reporting.  Host code only; the kernels live in kernels_*.cu.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/lbman3d.h"
#include "launch.h"
#include "solver_view.h"
#include "stats.h"
#include "tiles.h"

using namespace lbman;

namespace {

thread_local std::string g_err;

int fail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_err = buf;
    return code;
}

#define LB_CUDA(call)                                                                             \
    do {                                                                                          \
        cudaError_t e_ = (call);                                                                  \
        if (e_ != cudaSuccess)                                                                    \
            return fail(e_ == cudaErrorMemoryAllocation ? LBMAN_ERR_NOMEM : LBMAN_ERR_CUDA,       \
                        "%s:%d %s: %s", __FILE__, __LINE__, #call, cudaGetErrorString(e_));       \
    } while (0)

#define LB_TRY(expr)                  \
    do {                              \
        int s_ = (expr);              \
        if (s_ != LBMAN_OK) return s_; \
    } while (0)

struct Ops {
    decltype(&launch_qforce_f64) qforce;
    decltype(&launch_fused_f64) fused;
    decltype(&launch_lbm_f64) lbm;
    decltype(&launch_stream_only_f64) stream_only;
    decltype(&launch_lbm_aa_f64) lbm_aa;
    decltype(&launch_aa_pop_out_f64) aa_pop_out;
    decltype(&launch_swap_pairs_f64) swap_pairs;
    decltype(&launch_halo_merge_f64) halo_merge;
    decltype(&launch_feq_init_f64) feq_init;
    decltype(&launch_pop_in_f64) pop_in;
    decltype(&launch_pop_out_f64) pop_out;
    decltype(&launch_real_in_f64) real_in;
    decltype(&launch_real_out_f64) real_out;
    decltype(&launch_flow_reduce_f64) flow_reduce;
    decltype(&launch_energy_reduce_f64) energy_reduce;
    decltype(&launch_defects_f64) defects;
    decltype(&launch_seeded_init_f64) seeded_init;
    decltype(&launch_qsetup_f64) qsetup;
    decltype(&launch_active_force_f64) active_force;
    decltype(&launch_qpoint_f64) qpoint;
    decltype(&launch_point_force_f64) point_force;
    decltype(&launch_lbm_aa_point_f64) lbm_aa_point;
    decltype(&qforce_smem_f64) qforce_smem;
    decltype(&qforce_threads_f64) qforce_threads;
    decltype(&march_blocks_f64) march_blocks;
    decltype(&prepare_f64) prepare;
};

// QSUF: the suffix of the kernels that do not touch populations (FP16 storage
// computes in FP32)
#define LBMAN_OPS(SUF, QSUF)                                                                               \
    Ops {                                                                                              \
        launch_qforce_##SUF, launch_fused_##SUF, launch_lbm_##SUF, launch_stream_only_##SUF,           \
            launch_lbm_aa_##SUF, launch_aa_pop_out_##SUF, launch_swap_pairs_##SUF,                     \
            launch_halo_merge_##SUF,                                                                   \
            launch_feq_init_##SUF, launch_pop_in_##SUF, launch_pop_out_##SUF, launch_real_in_##SUF,    \
            launch_real_out_##SUF, launch_flow_reduce_##QSUF, launch_energy_reduce_##QSUF,             \
            launch_defects_##QSUF,                                                                     \
            launch_seeded_init_##SUF, launch_qsetup_##SUF, launch_active_force_##SUF,                  \
            launch_qpoint_##QSUF, launch_point_force_##QSUF, launch_lbm_aa_point_##SUF,                \
            qforce_smem_##SUF, qforce_threads_##SUF, march_blocks_##SUF, prepare_##SUF                 \
    }

const Ops kOps[3] = {LBMAN_OPS(f64, f64), LBMAN_OPS(f32, f32), LBMAN_OPS(f16, f32)};

// AnchoredQ (src/boundary_handler.h:232-251), evaluated on the host.
void anchored_q(const lbman_face& f, double out[5]) {
    if (f.qbc != LBMAN_Q_ANCHORING) {
        for (int k = 0; k < 5; ++k) out[k] = 0.0;
        return;
    }
    const double sin_sq_phi = 0.5 * (1.0 - std::cos(2.0 * f.phi));
    const double cos_sq_phi = 1.0 - sin_sq_phi;
    const double sin_phi_cos_phi = 0.5 * std::sin(2.0 * f.phi);
    const double sin_sq_th = 0.5 * (1.0 - std::cos(2.0 * f.theta));
    const double sin_th_cos_th = 0.5 * std::sin(2.0 * f.theta);
    const double S = f.s;
    out[0] = S * (cos_sq_phi * sin_sq_th - 1.0 / 3.0);
    out[1] = S * (sin_phi_cos_phi * sin_sq_th);
    out[2] = S * (std::cos(f.phi) * sin_th_cos_th);
    out[3] = S * (sin_sq_phi * sin_sq_th - 1.0 / 3.0);
    out[4] = S * (std::sin(f.phi) * sin_th_cos_th);
}

}  // namespace

namespace lbman {
// Error message for lbman_last_error() from other translation units.
void set_last_error(const char* msg) { g_err = msg; }

// params.h + BC configuration -> the kernels' SimParams.
void build_sim_params(const lbman_config& c, SimParams& P) {
    std::memset(&P, 0, sizeof(P));
    P.nx = c.nx; P.ny = c.ny; P.nz = c.nz;
    P.nxy = (int64_t)c.nx * c.ny;
    P.V = P.nxy * c.nz;
    P.zlo = 0;
    P.zhi = c.nz;
    P.c0 = 0;
    P.c1 = P.V;
    P.gbase = 0;
    P.DT = c.DT; P.kDensity = c.kDensity; P.L = c.L; P.A = c.A; P.B = c.B; P.C = c.C;
    P.LAMBDA = c.LAMBDA; P.GAMMA = c.GAMMA; P.ALPHA = c.ALPHA; P.MU = c.MU;
    // src/params.h:52-54
    P.omega = 1.0 - c.DT / c.TAUF;
    P.omega_prime = c.DT / c.TAUF;
    P.omega_forcing = 1.0 - c.DT / 2.0 / c.TAUF;
    P.upwind = c.advection == LBMAN_UPWIND;
    P.half_pop = c.precision == LBMAN_FP16;
    P.moving_any = 0;
    for (int k = 0; k < 6; ++k) {
        P.face[k].qbc = c.face[k].qbc;
        P.face[k].ubc = c.face[k].ubc;
        anchored_q(c.face[k], P.face[k].anchor);
        for (int j = 0; j < 3; ++j) P.face[k].uw[j] = c.face[k].ubc == LBMAN_U_MOVING ? c.face[k].uw[j] : 0.0;
        P.qper[k] = c.face[k].qbc == LBMAN_Q_PERIODIC;
        P.uper[k] = c.face[k].ubc == LBMAN_U_PERIODIC;
        if (c.face[k].ubc == LBMAN_U_MOVING) P.moving_any = 1;
    }
    fill_float_phys(P);
}
}  // namespace lbman

enum { F_PRE = 0, F_POST = 1, F_SWAP = 2 };

struct lbman_solver {
    lbman_config cfg;
    SimParams P;
    LaunchShape shape;
    int prec = LBMAN_FP64;
    int kernels = LBMAN_KERNELS_FUSED;
    int device = 0;
    size_t rbytes = 8, sbytes = 8;
    void* f[2] = {nullptr, nullptr};
    void* q[2] = {nullptr, nullptr};
    void* u[2] = {nullptr, nullptr};
    void* rho = nullptr;
    void* F = nullptr;
    // Point organisation (qpoint.cuh): steps run without the z-marching Q
    // kernel; pstress holds the stress between its two kernels.  A handle it
    // can step (point_able) names it by the shape it was created with.
    bool point = false, point_able = false;
    lbman_shape untuned{};
    void* pstress = nullptr;
    void* stress = nullptr;  // Sigma (5) and tau (3) of the two-phase Q stage, allocated on first use
    double* staging = nullptr;
    double* partials = nullptr;
    int red_G = 0;
    double* red_dev = nullptr;
    double* red_host = nullptr;
    void* upast = nullptr;
    int fcur = 0, qcur = 0, ucur = 0;
    // Layout of the populations in f[fcur]: F_PRE pre-collision (after an
    // upload or an odd in-place step), F_POST post-collision of the
    // two-buffer kernels (fused organisation), F_SWAP post-collision in the
    // in-place layout (after an even in-place step).  f[1] exists only once
    // the fused organisation has run.
    int fphase = 0;
    bool uploaded = false;
    // z-slab of a larger box (lbman_create_slab): owned planes [P.zlo, P.zhi)
    // of an allocation with two ghost planes on each side.  The flags order
    // the exchanges around the steps: the Q/u halo is fresh (exchanged since
    // the last step), the population halo of an odd step is in, and the
    // populations an odd step scattered into the ghost planes are still to
    // be merged by the neighbours.
    bool slab = false;
    int nz_global = 0, z_offset = 0;
    void* fstage = nullptr;  // F_OUT arrivals: 2 faces x 5 slots x nx*ny
    bool qu_fresh = false, fin_fresh = false, fout_pending = false;
    cudaEvent_t ev_ready = nullptr, ev_done = nullptr;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    int64_t steps = 0, launches = 0;
    int num_sms = 148;
    lbman::stats::Workspace* stats = nullptr;
    const Ops& ops() const { return kOps[prec]; }
};

namespace {

int set_device(lbman_solver* s) {
    LB_CUDA(cudaSetDevice(s->device));
    return LBMAN_OK;
}

int check_launch(lbman_solver* s, cudaError_t e, const char* what) {
    ++s->launches;
    if (e != cudaSuccess) return fail(LBMAN_ERR_CUDA, "%s launch failed: %s", what, cudaGetErrorString(e));
    return LBMAN_OK;
}


// z chunk giving several waves of blocks over the SMs, and at most 256
// planes (1024^3: 74 ms per step in 1024-plane chunks, 66 ms in 256).
int default_zchunk(int nx, int ny, int nz, int tcx, int tcy, int num_sms) {
    const long cols = (long)((nx + tcx - 1) / tcx) * ((ny + tcy - 1) / tcy);
    const long target = (long)num_sms * 8;
    long nchunks = (target + cols - 1) / cols;
    nchunks = std::max(1L, std::min(nchunks, (long)std::max(1, nz / 8)));
    nchunks = std::max(nchunks, (long)((nz + 255) / 256));
    return (int)((nz + nchunks - 1) / nchunks);
}

// Largest box (cells) an untuned AUTO handle steps with the point kernels
// (qpoint.cuh): they index 15 V in 32 bits.  Below that they were the faster
// ones at every size tried.  Whole steps on B200, z-marching kernels -> these:
//   FP64             32^3 67 -> 8 us, 256^3 2865 -> 2070 us
//   FP32, one point  64x256x256 slit 282 -> 243 us, 256^3 slit 981 -> 834 us,
//                    301x300x300 channel 2914 -> 1766 us
//   FP32, packed     240x160x165 350 -> 310 us, 256^3 909 -> 784 us, 512x512x256
//                    3470 -> 3162 us, 512^3 6918 -> 6423 us
//   FP16, packed     240x240x60 189 -> 161 us, 256^3 811 -> 704 us, 512x512x256
//                    3055 -> 2848 us
constexpr int64_t kPointCells = (((int64_t)1 << 31) - 1) / 15;

// FP64 boxes with z walls or anchoring (whose kernels carry every wall rule)
// form the body force in a kernel of its own above this size: 200^3 1485 us per
// step, 1533 us with the force formed by the LBM kernel.  All others form it
// there, a launch and the force's round trip less: FP64 200^3 1001 us for 1073,
// 256^3 2070 for 2216, 256^3 slit 2165 for 2343, 301x200x150 channel 1300 for
// 1333; FP32 256^3 slit 834 for 858.
constexpr int64_t kPointFusedCells = (int64_t)6 << 20;
bool force_apart(const SimParams& P) {
    bool general = !(P.qper[4] && P.qper[5] && P.uper[4] && P.uper[5]);
    for (const Face& f : P.face) general = general || f.qbc == Q_ANCHORING;
    return general && P.V > kPointFusedCells;
}

// Memory (words per cell) a handle must leave free when it takes the point
// kernels' scratch: the buffers it may ask for later (second population buffer,
// two-phase stress, snapshots, statistics), so that none of them fails for it.
constexpr int64_t kPointSpareWords = 48;

// Scratch of the point kernels: 9 row-stress words (FP32) or Sigma and tau
// (FP64) per cell.  A box that has no room for them keeps the z-marching kernels.
bool take_point(lbman_solver* s) {
    const size_t words = s->prec == LBMAN_FP64 ? 8 : 9;
    size_t free_bytes = 0, total = 0;
    if (!s->pstress && (cudaMemGetInfo(&free_bytes, &total) != cudaSuccess ||
                        (words + kPointSpareWords) * s->P.V * s->rbytes > free_bytes ||
                        cudaMalloc(&s->pstress, words * s->P.V * s->rbytes) != cudaSuccess)) {
        cudaGetLastError();
        s->pstress = nullptr;
    }
    return s->point = s->pstress != nullptr;
}

// The z-marching kernels from here on; the point kernels' scratch is given back.
void drop_point(lbman_solver* s) {
    s->point = false;
    cudaFree(s->pstress);
    s->pstress = nullptr;
}

// Default z-marching tile before any autotuning: the widest compiled tile
// up to 32 cells whose last partial tile pads x by at most 10% (wide rows
// keep the global stores of a block in full sectors); otherwise the one with
// the least work per output cell (threads per tile cell times the x and y
// padding).
LaunchShape default_shape(const lbman_config& c, int num_sms, const Ops& ops) {
    LaunchShape L;
    L.tile.pair = c.kernels == LBMAN_KERNELS_SPLIT_PAIR;
    if (c.tile_x > 0 && c.tile_y > 0) {
        L.tile.tcx = c.tile_x;
        L.tile.tcy = c.tile_y;
    } else if (L.tile.pair) {
        L.tile.tcx = 30;
        L.tile.tcy = 10;
    } else {
        double best = 1e30;
        int best_wide = -1;
        L.tile.tcx = 30;
        L.tile.tcy = 6;
        for (const auto& t : kTileList) {
            QTile q{t[0], t[1], 1};
            if (ops.qforce_smem(q) == 0) continue;  // not compiled for this precision
            const double padx = (double)((c.nx + t[0] - 1) / t[0] * t[0]) / c.nx;
            const double pady = (double)((c.ny + t[1] - 1) / t[1] * t[1]) / c.ny;
            const double cost = padx * pady * ops.qforce_threads(q) / (double)(t[0] * t[1]);
            // the widest tile up to one warp per row: 64-wide rows measured
            // slower (512^3: 5.3 ms Q stage at 64x6 against 4.4 ms at 32x8)
            if (padx <= 1.10 && t[0] <= 32 && t[0] > best_wide) {
                best_wide = t[0];
                L.tile.tcx = t[0];
                L.tile.tcy = t[1];
            }
            if (best_wide < 0 && cost < best - 1e-9) {
                best = cost;
                L.tile.tcx = t[0];
                L.tile.tcy = t[1];
            }
        }
        // among the 32-wide tiles, 32x8 (what the autotuner picks for the slit
        // and close to its 512^3 choice)
        const QTile q328{32, 8, 1};
        if (L.tile.tcx == 32 && ops.qforce_smem(q328) != 0) L.tile.tcy = 8;
    }
    L.qthreads = ops.qforce_threads(L.tile);
    // fixed z chunks giving several waves of blocks: measured on B200 the
    // autotuner picks them over the balanced one-wave schedule on every
    // workload (the pair kernel at 512^3: 6.7 ms balanced, 4.0 ms in 64-plane
    // chunks), so an untuned handle starts there
    L.tile.zc = c.zchunk > 0 ? c.zchunk : default_zchunk(c.nx, c.ny, c.nz, L.tile.tcx, L.tile.tcy, num_sms);
    L.num_sms = num_sms;
    return L;
}

int validate(const lbman_config& c) {
    if (c.nx < 1 || c.ny < 1 || c.nz < 1) return fail(LBMAN_ERR_ARG, "grid must be at least 1x1x1");
    const double V = (double)c.nx * c.ny * c.nz;
    if (V >= 2147483648.0) return fail(LBMAN_ERR_UNSUPPORTED, "grids of 2^31 cells or more are not supported");
    if (c.precision < LBMAN_FP64 || c.precision > LBMAN_FP16) return fail(LBMAN_ERR_ARG, "bad precision");
    if (c.advection != LBMAN_CENTRED && c.advection != LBMAN_UPWIND) return fail(LBMAN_ERR_ARG, "bad advection");
    if (c.kernels < LBMAN_KERNELS_AUTO || c.kernels > LBMAN_KERNELS_SPLIT_PAIR) return fail(LBMAN_ERR_ARG, "bad kernels");
    if (c.kernels == LBMAN_KERNELS_SPLIT_PAIR && (c.precision == LBMAN_FP64 || (c.nx & 3) != 0))
        return fail(LBMAN_ERR_ARG, "LBMAN_KERNELS_SPLIT_PAIR needs FP32 or FP16 precision and nx a multiple of 4");
    if (!(c.TAUF > 0.0) || !(c.DT > 0.0) || !(c.kDensity > 0.0)) return fail(LBMAN_ERR_ARG, "TAUF, DT, kDensity must be > 0");
    for (int k = 0; k < 6; ++k) {
        const lbman_face& f = c.face[k];
        if (f.qbc < LBMAN_Q_PERIODIC || f.qbc > LBMAN_Q_ANCHORING) return fail(LBMAN_ERR_ARG, "face %d: bad Q tag", k);
        if (f.ubc < LBMAN_U_PERIODIC || f.ubc > LBMAN_U_SPECULAR) return fail(LBMAN_ERR_ARG, "face %d: bad velocity tag", k);
    }
    for (int ax = 0; ax < 3; ++ax) {
        const bool lo = c.face[2 * ax].ubc == LBMAN_U_PERIODIC, hi = c.face[2 * ax + 1].ubc == LBMAN_U_PERIODIC;
        if (lo != hi)
            return fail(LBMAN_ERR_ARG,
                        "axis %c: the velocity tag is periodic on one face only; streaming across such an axis "
                        "has two writers per population in the reference and is not supported",
                        "xyz"[ax]);
    }
    if (c.tile_x < 0 || c.tile_y < 0 || c.zchunk < 0 || c.threads < 0) return fail(LBMAN_ERR_ARG, "bad launch shape");
    return LBMAN_OK;
}

int stage_in_real(lbman_solver* s, const double* host, void* dst, int64_t n) {
    if (s->prec == LBMAN_FP64) {
        LB_CUDA(cudaMemcpyAsync(dst, host, n * sizeof(double), cudaMemcpyHostToDevice, s->stream));
        return LBMAN_OK;
    }
    LB_CUDA(cudaMemcpyAsync(s->staging, host, n * sizeof(double), cudaMemcpyHostToDevice, s->stream));
    return check_launch(s, s->ops().real_in(s->staging, dst, n, s->stream), "real_in");
}

int stage_out_real(lbman_solver* s, const void* src, double* host, int64_t n) {
    if (s->prec == LBMAN_FP64) {
        LB_CUDA(cudaMemcpyAsync(host, src, n * sizeof(double), cudaMemcpyDeviceToHost, s->stream));
        return LBMAN_OK;
    }
    LB_TRY(check_launch(s, s->ops().real_out(src, s->staging, n, s->stream), "real_out"));
    LB_CUDA(cudaMemcpyAsync(host, s->staging, n * sizeof(double), cudaMemcpyDeviceToHost, s->stream));
    return LBMAN_OK;
}

void* vptr(void* base, int64_t off_elems, size_t esize) { return (char*)base + off_elems * (int64_t)esize; }

}  // namespace

namespace lbman {
int validate_config(const lbman_config& c) { return validate(c); }
}  // namespace lbman

extern "C" {

int lbman_abi_version(void) { return LBMAN_ABI_VERSION; }

const char* lbman_last_error(void) { return g_err.c_str(); }

const char* lbman_status_string(int status) {
    switch (status) {
        case LBMAN_OK: return "ok";
        case LBMAN_ERR_ARG: return "invalid argument";
        case LBMAN_ERR_CUDA: return "CUDA error";
        case LBMAN_ERR_DIVERGED: return "simulation diverged (NaN in mass or momentum)";
        case LBMAN_ERR_TIMEOUT: return "bounded device wait timed out";
        case LBMAN_ERR_STATE: return "call out of order";
        case LBMAN_ERR_UNSUPPORTED: return "unsupported configuration";
        case LBMAN_ERR_NOMEM: return "device allocation failed";
        default: return "unknown status";
    }
}

int lbman_config_init(lbman_config* c) {
    if (!c) return fail(LBMAN_ERR_ARG, "null config");
    std::memset(c, 0, sizeof(*c));
    // src/params.h:14-112
    c->nx = 20; c->ny = 100; c->nz = 100;
    c->DT = 1.0; c->kDensity = 1.0; c->TAUF = 2.5 * 1.0;
    c->L = 0.06; c->A = 0.0; c->B = -0.3; c->C = 0.3;
    c->LAMBDA = 0.3; c->GAMMA = 0.34; c->ALPHA = 0.023; c->MU = 0.0;
    c->advection = LBMAN_CENTRED;
    // SimBC = SlitNoSlipConfig (src/sim_config.h:37-48)
    for (int k = 0; k < 6; ++k) { c->face[k].qbc = LBMAN_Q_PERIODIC; c->face[k].ubc = LBMAN_U_PERIODIC; }
    c->face[0].qbc = c->face[1].qbc = LBMAN_Q_NEUMANN;
    c->face[0].ubc = c->face[1].ubc = LBMAN_U_NOSLIP;
    c->precision = LBMAN_FP64;
    c->kernels = LBMAN_KERNELS_AUTO;
    c->device = 0;
    return LBMAN_OK;
}

int lbman_device_info(int device, char* buf, size_t len) {
    if (!buf || len == 0) return fail(LBMAN_ERR_ARG, "null buffer");
    cudaDeviceProp p;
    LB_CUDA(cudaGetDeviceProperties(&p, device));
    size_t fr = 0, tot = 0;
    LB_CUDA(cudaSetDevice(device));
    LB_CUDA(cudaMemGetInfo(&fr, &tot));
    snprintf(buf, len,
             "GPU\n       using device: %d\n               name: %s\n    multiprocessors: %d\n"
             " compute capability: %d.%d\n      global memory: %.1f MiB\n        free memory: %.1f MiB\n",
             device, p.name, p.multiProcessorCount, p.major, p.minor, tot / 1048576.0, fr / 1048576.0);
    return LBMAN_OK;
}

int lbman_create(const lbman_config* cfg, lbman_solver** out) {
    if (!cfg || !out) return fail(LBMAN_ERR_ARG, "null argument");
    *out = nullptr;
    LB_TRY(validate(*cfg));
    lbman_solver* s = new lbman_solver();
    s->cfg = *cfg;
    s->device = cfg->device;
    s->prec = cfg->precision;
    // Measured on B200: the split organisations (Q+force kernel, then the
    // LBM kernel) outrun the one-kernel step for every workload and tile
    // tried, and the two-points-per-thread Q kernel is the faster of the two
    // where its 30-wide tiles pad x by at most 10% (512^3: 19.3 against 18.2
    // GLUPS untuned); so those are the defaults until lbman_autotune says
    // otherwise.  The point kernels have no tiles, but take their arithmetic
    // (one point or packed) from the same rule, so that a box has the same bits
    // with and without them.
    int kern = cfg->kernels;
    if (kern == LBMAN_KERNELS_AUTO) {
        const bool pair_fits = cfg->precision != LBMAN_FP64 && cfg->nx % 4 == 0 && cfg->tile_x == 0 &&
                               cfg->tile_y == 0 && (double)((cfg->nx + 29) / 30 * 30) <= 1.10 * cfg->nx;
        kern = pair_fits ? LBMAN_KERNELS_SPLIT_PAIR : LBMAN_KERNELS_SPLIT;
    }
    s->kernels = kern;
    s->rbytes = s->prec == LBMAN_FP64 ? 8 : 4;
    s->sbytes = s->prec == LBMAN_FP64 ? 8 : (s->prec == LBMAN_FP32 ? 4 : 2);
    auto bail = [&](int code) {
        lbman_destroy(s);
        return code;
    };
    if (int st = set_device(s)) return bail(st);
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, s->device) != cudaSuccess)
        return bail(fail(LBMAN_ERR_CUDA, "cudaGetDeviceProperties failed"));
    if (prop.major < 10) return bail(fail(LBMAN_ERR_UNSUPPORTED, "this library targets sm_100a (B200); device is sm_%d%d", prop.major, prop.minor));
    s->num_sms = prop.multiProcessorCount;

    build_sim_params(*cfg, s->P);
    lbman_config resolved = *cfg;
    resolved.kernels = kern;
    s->shape = default_shape(resolved, s->num_sms, s->ops());
    const size_t smem = s->ops().qforce_smem(s->shape.tile);
    if (smem == 0)
        return bail(fail(LBMAN_ERR_ARG, "tile %dx%d is not compiled for this precision (compiled: 30x6, 32x6, "
                                        "14x14, and for FP32/FP16 also 30x14, 62x6)",
                         s->shape.tile.tcx, s->shape.tile.tcy));
    if (smem > (size_t)prop.sharedMemPerBlockOptin)
        return bail(fail(LBMAN_ERR_ARG, "tile %dx%d needs %zu B of shared memory (max %zu)", s->shape.tile.tcx,
                         s->shape.tile.tcy, smem, (size_t)prop.sharedMemPerBlockOptin));
    if (cfg->threads > 0 && cfg->threads != s->shape.qthreads)
        return bail(fail(LBMAN_ERR_ARG, "tile %dx%d runs %d threads per block", s->shape.tile.tcx,
                         s->shape.tile.tcy, s->shape.qthreads));
    if (cudaError_t e = s->ops().prepare(prop.sharedMemPerBlockOptin))
        return bail(fail(LBMAN_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e)));

    const int64_t V = s->P.V;
    auto alloc = [&](void** p, size_t bytes) -> int {
        cudaError_t e = cudaMalloc(p, bytes);
        if (e != cudaSuccess) return fail(LBMAN_ERR_NOMEM, "cudaMalloc(%zu) failed: %s", bytes, cudaGetErrorString(e));
        return LBMAN_OK;
    };
    // one population buffer: the split organisations stream in place
    if (int st = alloc(&s->f[0], 15 * V * s->sbytes)) return bail(st);
    for (int b = 0; b < 2; ++b) {
        if (int st = alloc(&s->q[b], 5 * V * s->rbytes)) return bail(st);
        if (int st = alloc(&s->u[b], 3 * V * s->rbytes)) return bail(st);
    }
    s->point_able = cfg->kernels == LBMAN_KERNELS_AUTO && cfg->tile_x == 0 && cfg->tile_y == 0 && cfg->zchunk == 0 &&
                    V <= kPointCells;
    s->untuned = {kern, s->shape.tile.tcx, s->shape.tile.tcy, s->shape.tile.zc, 0, 0.0, 0};
    if (s->point_able) take_point(s);
    if (int st = alloc(&s->rho, V * s->rbytes)) return bail(st);
    if (int st = alloc(&s->F, 3 * V * s->rbytes)) return bail(st);
    // FP64 host staging too: downloads of an in-place-layout state gather
    // into it
    if (int st = alloc((void**)&s->staging, V * sizeof(double))) return bail(st);
    s->red_G = (int)std::min<int64_t>((V + 255) / 256, (int64_t)s->num_sms * 8);
    if (int st = alloc((void**)&s->partials, (size_t)s->red_G * 8 * sizeof(double))) return bail(st);
    if (int st = alloc((void**)&s->red_dev, 16 * sizeof(double))) return bail(st);
    if (cudaMallocHost((void**)&s->red_host, 16 * sizeof(double)) != cudaSuccess)
        return bail(fail(LBMAN_ERR_NOMEM, "cudaMallocHost failed"));
    if (cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) != cudaSuccess)
        return bail(fail(LBMAN_ERR_CUDA, "cudaStreamCreate failed"));
    s->own_stream = true;
    *out = s;
    return LBMAN_OK;
}

int lbman_destroy(lbman_solver* s) {
    if (!s) return LBMAN_OK;
    cudaSetDevice(s->device);
    if (s->stream) cudaStreamSynchronize(s->stream);
    for (int b = 0; b < 2; ++b) { cudaFree(s->f[b]); cudaFree(s->q[b]); cudaFree(s->u[b]); }
    cudaFree(s->rho); cudaFree(s->F); cudaFree(s->staging); cudaFree(s->partials); cudaFree(s->red_dev);
    cudaFree(s->upast); cudaFree(s->stress); cudaFree(s->pstress); cudaFree(s->fstage);
    if (s->ev_ready) cudaEventDestroy(s->ev_ready);
    if (s->ev_done) cudaEventDestroy(s->ev_done);
    lbman::stats::destroy(s->stats);
    if (s->red_host) cudaFreeHost(s->red_host);
    if (s->own_stream && s->stream) cudaStreamDestroy(s->stream);
    delete s;
    return LBMAN_OK;
}

int lbman_set_stream(lbman_solver* s, void* stream) {
    if (!s) return fail(LBMAN_ERR_ARG, "null solver");
    LB_TRY(set_device(s));
    LB_CUDA(cudaStreamSynchronize(s->stream));
    if (s->own_stream) cudaStreamDestroy(s->stream);
    s->stream = (cudaStream_t)stream;
    s->own_stream = false;
    return LBMAN_OK;
}

int lbman_synchronize(lbman_solver* s) {
    if (!s) return fail(LBMAN_ERR_ARG, "null solver");
    LB_TRY(set_device(s));
    LB_CUDA(cudaStreamSynchronize(s->stream));
    return LBMAN_OK;
}

int lbman_upload(lbman_solver* s, const double* rho, const double* u3, const double* q5, const double* f15,
                 const double* force3) {
    if (!s || !rho || !u3 || !q5) return fail(LBMAN_ERR_ARG, "rho, u and q are required");
    LB_TRY(set_device(s));
    // host arrays hold the owned cells [c0, c1) (the whole box unless a slab)
    const int64_t V = s->P.V, c0 = s->P.c0, Vo = s->P.c1 - s->P.c0;
    LB_TRY(stage_in_real(s, rho, vptr(s->rho, c0, s->rbytes), Vo));
    for (int k = 0; k < 3; ++k) LB_TRY(stage_in_real(s, u3 + k * Vo, vptr(s->u[s->ucur], k * V + c0, s->rbytes), Vo));
    for (int k = 0; k < 5; ++k) LB_TRY(stage_in_real(s, q5 + k * Vo, vptr(s->q[s->qcur], k * V + c0, s->rbytes), Vo));
    if (force3) {
        for (int k = 0; k < 3; ++k) LB_TRY(stage_in_real(s, force3 + k * Vo, vptr(s->F, k * V + c0, s->rbytes), Vo));
    } else {
        LB_CUDA(cudaMemsetAsync(s->F, 0, 3 * V * s->rbytes, s->stream));
    }
    if (f15) {
        for (int j = 0; j < 15; ++j) {
            if (s->prec == LBMAN_FP64) {
                LB_CUDA(cudaMemcpyAsync(vptr(s->f[s->fcur], j * V + c0, 8), f15 + j * Vo, Vo * 8, cudaMemcpyHostToDevice,
                                        s->stream));
            } else {
                LB_CUDA(cudaMemcpyAsync(s->staging + c0, f15 + j * Vo, Vo * 8, cudaMemcpyHostToDevice, s->stream));
                LB_TRY(check_launch(s, s->ops().pop_in(s->P, s->staging, s->f[s->fcur], j, s->stream), "pop_in"));
            }
        }
    } else {
        LB_TRY(check_launch(s, s->ops().feq_init(s->P, s->rho, s->u[s->ucur], s->f[s->fcur], s->stream), "feq_init"));
    }
    LB_CUDA(cudaStreamSynchronize(s->stream));
    s->uploaded = true;
    s->fphase = F_PRE;
    s->steps = 0;
    s->qu_fresh = s->fin_fresh = s->fout_pending = false;
    return LBMAN_OK;
}

}  // extern "C"

namespace lbman {

int solver_view(lbman_solver* s, SolverView* v) {
    if (!s || !v) return fail(LBMAN_ERR_ARG, "null argument");
    v->prec = s->prec;
    v->nx = s->P.nx;
    v->ny = s->P.ny;
    v->nz = s->P.nz;
    v->V = s->P.V;
    v->rho = s->rho;
    v->u = s->u[s->ucur];
    v->q = s->q[s->qcur];
    v->stream = s->stream;
    v->uploaded = s->uploaded;
    return LBMAN_OK;
}

int solver_reset_populations(lbman_solver* s) {
    if (!s) return fail(LBMAN_ERR_ARG, "null solver");
    if (!s->uploaded) return fail(LBMAN_ERR_STATE, "no state to rebuild populations from");
    LB_TRY(set_device(s));
    LB_TRY(check_launch(s, s->ops().feq_init(s->P, s->rho, s->u[s->ucur], s->f[s->fcur], s->stream), "feq_init"));
    s->fphase = F_PRE;
    return LBMAN_OK;
}

int solver_set_state(lbman_solver* s, const void* rho, const void* u3, const void* q5) {
    if (!s || !rho || !u3 || !q5) return fail(LBMAN_ERR_ARG, "null argument");
    LB_TRY(set_device(s));
    const int64_t V = s->P.V;
    LB_CUDA(cudaMemcpyAsync(s->rho, rho, V * s->rbytes, cudaMemcpyDeviceToDevice, s->stream));
    LB_CUDA(cudaMemcpyAsync(s->u[s->ucur], u3, 3 * V * s->rbytes, cudaMemcpyDeviceToDevice, s->stream));
    LB_CUDA(cudaMemcpyAsync(s->q[s->qcur], q5, 5 * V * s->rbytes, cudaMemcpyDeviceToDevice, s->stream));
    LB_CUDA(cudaMemsetAsync(s->F, 0, 3 * V * s->rbytes, s->stream));
    s->uploaded = true;
    s->steps = 0;
    return solver_reset_populations(s);
}

}  // namespace lbman

extern "C" {

int lbman_init_seeded(lbman_solver* s, uint64_t seed, double S0, double sigma) {
    if (!s) return fail(LBMAN_ERR_ARG, "null solver");
    LB_TRY(set_device(s));
    LB_TRY(check_launch(s, s->ops().seeded_init(s->P, seed, S0, sigma, s->rho, s->u[s->ucur], s->q[s->qcur], s->F, s->stream),
                        "seeded_init"));
    LB_TRY(check_launch(s, s->ops().feq_init(s->P, s->rho, s->u[s->ucur], s->f[s->fcur], s->stream), "feq_init"));
    LB_CUDA(cudaStreamSynchronize(s->stream));
    s->uploaded = true;
    s->fphase = F_PRE;
    s->steps = 0;
    s->qu_fresh = s->fin_fresh = s->fout_pending = false;
    return LBMAN_OK;
}

int lbman_download(lbman_solver* s, double* rho, double* u3, double* q5, double* f15, double* force3) {
    if (!s) return fail(LBMAN_ERR_ARG, "null solver");
    if (!s->uploaded) return fail(LBMAN_ERR_STATE, "download before upload");
    if (s->slab && s->fout_pending)
        return fail(LBMAN_ERR_STATE, "exchange LBMAN_HALO_F_OUT after an odd step before downloading a slab");
    if (s->slab && f15 && s->fphase == F_SWAP && !s->fin_fresh)
        return fail(LBMAN_ERR_STATE, "exchange LBMAN_HALO_F_IN before downloading a slab's populations here");
    LB_TRY(set_device(s));
    const int64_t V = s->P.V, c0 = s->P.c0, Vo = s->P.c1 - s->P.c0;
    if (rho) LB_TRY(stage_out_real(s, vptr(s->rho, c0, s->rbytes), rho, Vo));
    if (u3)
        for (int k = 0; k < 3; ++k) LB_TRY(stage_out_real(s, vptr(s->u[s->ucur], k * V + c0, s->rbytes), u3 + k * Vo, Vo));
    if (q5)
        for (int k = 0; k < 5; ++k) LB_TRY(stage_out_real(s, vptr(s->q[s->qcur], k * V + c0, s->rbytes), q5 + k * Vo, Vo));
    if (force3)
        for (int k = 0; k < 3; ++k) LB_TRY(stage_out_real(s, vptr(s->F, k * V + c0, s->rbytes), force3 + k * Vo, Vo));
    if (f15) {
        const void* src = s->f[s->fcur];
        if (s->fphase == F_POST) {  // stream the stored f* into the spare buffer
            LB_TRY(check_launch(s, s->ops().stream_only(s->P, s->f[s->fcur], s->f[1 - s->fcur], s->rho, s->stream), "stream_only"));
            src = s->f[1 - s->fcur];
        }
        for (int j = 0; j < 15; ++j) {
            if (s->fphase == F_SWAP) {  // the odd step's gather of direction j
                if (!s->staging) return fail(LBMAN_ERR_STATE, "no staging buffer");
                LB_TRY(check_launch(s, s->ops().aa_pop_out(s->P, src, s->rho, s->staging, j, s->stream), "aa_pop_out"));
                LB_CUDA(cudaMemcpyAsync(f15 + j * Vo, s->staging + c0, Vo * 8, cudaMemcpyDeviceToHost, s->stream));
            } else if (s->prec == LBMAN_FP64) {
                LB_CUDA(cudaMemcpyAsync(f15 + j * Vo, vptr((void*)src, j * V + c0, 8), Vo * 8, cudaMemcpyDeviceToHost,
                                        s->stream));
            } else {
                LB_TRY(check_launch(s, s->ops().pop_out(s->P, src, s->staging, j, s->stream), "pop_out"));
                LB_CUDA(cudaMemcpyAsync(f15 + j * Vo, s->staging + c0, Vo * 8, cudaMemcpyDeviceToHost, s->stream));
            }
        }
    }
    LB_CUDA(cudaStreamSynchronize(s->stream));
    return LBMAN_OK;
}

// The second population buffer of the fused (two-buffer) organisation.
static int ensure_f1(lbman_solver* s) {
    if (!s->f[1]) {
        cudaError_t e = cudaMalloc(&s->f[1], 15 * s->P.V * s->sbytes);
        if (e != cudaSuccess) {
            cudaGetLastError();
            s->f[1] = nullptr;
            return fail(LBMAN_ERR_NOMEM, "cudaMalloc of the second population buffer failed: %s", cudaGetErrorString(e));
        }
    }
    // the buffers alternate; f[fcur] must be the one in use
    return LBMAN_OK;
}

// A two-buffer post-collision state is put in the in-place layout.
static int aa_layout(lbman_solver* s) {
    if (s->fphase == F_POST) {
        LB_TRY(check_launch(s, s->ops().swap_pairs(s->P, s->f[s->fcur], s->stream), "swap_pairs"));
        s->fphase = F_SWAP;
    }
    return LBMAN_OK;
}

// In-place LBM step (AA pattern): even from F_PRE, odd from F_SWAP.
static int aa_step(lbman_solver* s, bool last) {
    const Ops& o = s->ops();
    LB_TRY(aa_layout(s));
    const bool odd = s->fphase == F_SWAP;
    LB_TRY(check_launch(s, o.lbm_aa(s->P, odd, last, s->f[s->fcur], s->F, s->rho, s->u[s->ucur], s->stream), "lbm_aa"));
    s->fphase = odd ? F_PRE : F_SWAP;
    return LBMAN_OK;
}

// The Q stage: Q_new, and the body force in s->F (force: formed here rather
// than by the LBM step that follows).
static int q_stage(lbman_solver* s, bool force) {
    const Ops& o = s->ops();
    if (s->point) {
        const bool pair = s->kernels == LBMAN_KERNELS_SPLIT_PAIR;
        LB_TRY(check_launch(s, o.qpoint(s->P, pair, s->num_sms, s->q[s->qcur], s->u[s->ucur], s->q[1 - s->qcur],
                                        s->pstress, s->F, s->stream),
                            "qpoint"));
        if (force)
            LB_TRY(check_launch(s, o.point_force(s->P, pair, s->num_sms, s->q[1 - s->qcur], s->pstress, s->u[s->ucur], s->F,
                                              s->stream),
                                "point_force"));
    } else {
        LB_TRY(check_launch(s, o.qforce(s->P, s->shape, s->q[s->qcur], s->u[s->ucur], s->q[1 - s->qcur], s->F, s->stream),
                            "qforce"));
    }
    s->qcur ^= 1;
    return LBMAN_OK;
}

static int one_step(lbman_solver* s, bool last) {
    const Ops& o = s->ops();
    if (s->kernels == LBMAN_KERNELS_FUSED) {
        LB_TRY(ensure_f1(s));
        if (s->fphase == F_SWAP) {  // back to the two-buffer layout
            LB_TRY(check_launch(s, o.swap_pairs(s->P, s->f[s->fcur], s->stream), "swap_pairs"));
            s->fphase = F_POST;
        }
        const bool first = s->fphase == F_PRE;
        LB_TRY(check_launch(s,
                            o.fused(s->P, s->shape, first, s->q[s->qcur], s->u[s->ucur], s->q[1 - s->qcur],
                                    s->u[1 - s->ucur], s->f[s->fcur], s->f[1 - s->fcur], s->rho,
                                    last ? s->F : nullptr, last, s->stream),
                            "fused step"));
        s->qcur ^= 1;
        s->ucur ^= 1;
        s->fcur ^= 1;
        s->fphase = F_POST;
    } else if (s->point && (s->prec != LBMAN_FP64 || !force_apart(s->P))) {
        LB_TRY(q_stage(s, false));
        LB_TRY(aa_layout(s));
        const bool odd = s->fphase == F_SWAP;
        LB_TRY(check_launch(s, o.lbm_aa_point(s->P, s->kernels == LBMAN_KERNELS_SPLIT_PAIR, s->num_sms, odd, last,
                                              s->f[s->fcur], s->q[s->qcur], s->pstress, s->F, s->rho, s->u[s->ucur],
                                              s->stream),
                            "lbm_aa_point"));
        s->fphase = odd ? F_PRE : F_SWAP;
    } else {
        LB_TRY(q_stage(s, true));
        LB_TRY(aa_step(s, last));
    }
    ++s->steps;
    return LBMAN_OK;
}

int lbman_step(lbman_solver* s, int nsteps) {
    if (!s || nsteps < 0) return fail(LBMAN_ERR_ARG, "bad arguments");
    if (!s->uploaded) return fail(LBMAN_ERR_STATE, "step before upload");
    if (s->slab)
        return fail(LBMAN_ERR_STATE, "a slab steps through lbman_qtensor_step and lbman_lbm_step with halo exchanges");
    LB_TRY(set_device(s));
    for (int n = 0; n < nsteps; ++n) LB_TRY(one_step(s, n == nsteps - 1));
    return LBMAN_OK;
}

int lbman_qtensor_step(lbman_solver* s) {
    if (!s) return fail(LBMAN_ERR_ARG, "null solver");
    if (!s->uploaded) return fail(LBMAN_ERR_STATE, "step before upload");
    if (s->slab && (!s->qu_fresh || s->fout_pending))
        return fail(LBMAN_ERR_STATE, s->fout_pending ? "exchange LBMAN_HALO_F_OUT after the odd LBM step first"
                                                     : "exchange LBMAN_HALO_QU before the Q stage of a slab");
    LB_TRY(set_device(s));
    LB_TRY(q_stage(s, true));
    s->qu_fresh = false;
    return LBMAN_OK;
}

static int ensure_stress(lbman_solver* s) {
    if (!s->stress) LB_CUDA(cudaMalloc(&s->stress, 8 * s->P.V * s->rbytes));
    return LBMAN_OK;
}

int lbman_qtensor_setup(lbman_solver* s) {
    if (!s) return fail(LBMAN_ERR_ARG, "null solver");
    if (!s->uploaded) return fail(LBMAN_ERR_STATE, "step before upload");
    if (s->slab) return fail(LBMAN_ERR_UNSUPPORTED, "the two-phase Q stage is not available on slabs");
    LB_TRY(set_device(s));
    LB_TRY(ensure_stress(s));
    const int64_t V = s->P.V;
    LB_TRY(check_launch(s, s->ops().qsetup(s->P, s->q[s->qcur], s->u[s->ucur], s->q[1 - s->qcur], s->stress,
                                           vptr(s->stress, 5 * V, s->rbytes), s->F, s->stream),
                        "qsetup"));
    s->qcur ^= 1;
    return LBMAN_OK;
}

int lbman_active_force(lbman_solver* s) {
    if (!s) return fail(LBMAN_ERR_ARG, "null solver");
    if (!s->uploaded) return fail(LBMAN_ERR_STATE, "step before upload");
    if (s->slab) return fail(LBMAN_ERR_UNSUPPORTED, "the two-phase Q stage is not available on slabs");
    if (!s->stress) return fail(LBMAN_ERR_STATE, "no stress: call lbman_qtensor_setup or lbman_upload_stress first");
    LB_TRY(set_device(s));
    const int64_t V = s->P.V;
    LB_TRY(check_launch(s, s->ops().active_force(s->P, s->q[s->qcur], s->stress, vptr(s->stress, 5 * V, s->rbytes),
                                                 s->u[s->ucur], s->F, s->stream),
                        "active_force"));
    return LBMAN_OK;
}

int lbman_upload_stress(lbman_solver* s, const double* sigma5, const double* tau3) {
    if (!s || !sigma5 || !tau3) return fail(LBMAN_ERR_ARG, "null argument");
    LB_TRY(set_device(s));
    LB_TRY(ensure_stress(s));
    const int64_t V = s->P.V;
    for (int k = 0; k < 5; ++k) LB_TRY(stage_in_real(s, sigma5 + k * V, vptr(s->stress, k * V, s->rbytes), V));
    for (int k = 0; k < 3; ++k) LB_TRY(stage_in_real(s, tau3 + k * V, vptr(s->stress, (5 + k) * V, s->rbytes), V));
    LB_CUDA(cudaStreamSynchronize(s->stream));
    return LBMAN_OK;
}

int lbman_download_stress(lbman_solver* s, double* sigma5, double* tau3) {
    if (!s) return fail(LBMAN_ERR_ARG, "null solver");
    if (!s->stress) return fail(LBMAN_ERR_STATE, "no stress: call lbman_qtensor_setup first");
    LB_TRY(set_device(s));
    const int64_t V = s->P.V;
    if (sigma5) for (int k = 0; k < 5; ++k) LB_TRY(stage_out_real(s, vptr(s->stress, k * V, s->rbytes), sigma5 + k * V, V));
    if (tau3) for (int k = 0; k < 3; ++k) LB_TRY(stage_out_real(s, vptr(s->stress, (5 + k) * V, s->rbytes), tau3 + k * V, V));
    LB_CUDA(cudaStreamSynchronize(s->stream));
    return LBMAN_OK;
}

int lbman_lbm_step(lbman_solver* s) {
    if (!s) return fail(LBMAN_ERR_ARG, "null solver");
    if (!s->uploaded) return fail(LBMAN_ERR_STATE, "step before upload");
    const bool odd = s->fphase == F_SWAP;
    if (s->slab && (s->fout_pending || (odd && !s->fin_fresh)))
        return fail(LBMAN_ERR_STATE, s->fout_pending ? "exchange LBMAN_HALO_F_OUT after the odd LBM step first"
                                                     : "exchange LBMAN_HALO_F_IN before an odd LBM step of a slab");
    LB_TRY(set_device(s));
    LB_TRY(aa_step(s, true));
    if (s->slab) {
        s->qu_fresh = s->fin_fresh = false;
        s->fout_pending = odd;
    }
    return LBMAN_OK;
}

int lbman_reduce(lbman_solver* s, int flags, lbman_diag* out) {
    if (!s || !out) return fail(LBMAN_ERR_ARG, "null argument");
    if (!s->uploaded) return fail(LBMAN_ERR_STATE, "reduce before upload");
    LB_TRY(set_device(s));
    const int64_t V = s->P.V;
    const int G = s->red_G;
    const Ops& o = s->ops();
    std::memset(out, 0, sizeof(*out));
    out->defect_faces = -1;
    if (flags & LBMAN_DIAG_FLOW) {
        if (!s->upast) {
            LB_CUDA(cudaMalloc(&s->upast, 3 * V * s->rbytes));
            LB_CUDA(cudaMemsetAsync(s->upast, 0, 3 * V * s->rbytes, s->stream));
        }
        LB_TRY(check_launch(s, o.flow_reduce(s->P, s->rho, s->u[s->ucur], s->upast, s->partials, G, s->stream), "flow_reduce"));
        LB_TRY(check_launch(s, launch_fold(s->partials, G, 8, 1, s->red_dev, s->stream), "fold"));
    }
    if ((flags & LBMAN_DIAG_ENERGY) && s->slab && !s->qu_fresh)
        return fail(LBMAN_ERR_STATE, "the free energy of a slab needs a fresh LBMAN_HALO_QU exchange");
    if (flags & LBMAN_DIAG_ENERGY) {
        LB_TRY(check_launch(s, o.energy_reduce(s->P, s->q[s->qcur], s->partials, G, s->stream), "energy_reduce"));
        LB_TRY(check_launch(s, launch_fold(s->partials, G, 1, 0, s->red_dev + 8, s->stream), "fold"));
    }
    // a slab's plaquettes across its faces need the neighbour's director:
    // not counted
    const bool defects = (flags & LBMAN_DIAG_DEFECTS) && !s->slab && s->P.nx >= 2 && s->P.ny >= 2 && s->P.nz >= 2;
    if (defects) {
        LB_TRY(check_launch(s, o.defects(s->P, s->q[s->qcur], nullptr, (unsigned long long*)(s->red_dev + 9), s->stream),
                            "defects"));
    }
    LB_CUDA(cudaMemcpyAsync(s->red_host, s->red_dev, 10 * sizeof(double), cudaMemcpyDeviceToHost, s->stream));
    LB_CUDA(cudaStreamSynchronize(s->stream));
    const double* r = s->red_host;
    if (flags & LBMAN_DIAG_FLOW) {
        out->mass = r[0]; out->px = r[1]; out->py = r[2]; out->pz = r[3];
        out->kinetic_energy = r[4]; out->rel_change_num = r[5]; out->rel_change_den = r[6]; out->umax2 = r[7];
        out->nan_detected = std::isnan(r[0]) || std::isnan(r[1]) || std::isnan(r[2]) || std::isnan(r[3]);
    }
    if (flags & LBMAN_DIAG_ENERGY) out->free_energy = r[8];
    if (defects) std::memcpy(&out->defect_faces, r + 9, sizeof(int64_t));  // an integer count
    if (out->nan_detected) return fail(LBMAN_ERR_DIVERGED, "NaN in the global mass or momentum");
    return LBMAN_OK;
}

namespace {

int stats_ready(lbman_solver* s, int nbins) {
    if (!s->uploaded) return fail(LBMAN_ERR_STATE, "statistics before upload");
    if (s->slab) return fail(LBMAN_ERR_UNSUPPORTED, "statistics of a slab: download the slabs and assemble the box");
    if (nbins < 1 || nbins > lbman::stats::kMaxBins)
        return fail(LBMAN_ERR_ARG, "nbins must be in [1, %d]", lbman::stats::kMaxBins);
    LB_TRY(set_device(s));
    if (!s->stats) s->stats = lbman::stats::create(s->P.nx, s->P.ny, s->P.nz, s->prec == LBMAN_FP64, s->num_sms);
    return LBMAN_OK;
}

int stats_status(int code, const char* what) {
    if (code == 0) return LBMAN_OK;
    const int st = lbman::stats::is_nomem(code) ? LBMAN_ERR_NOMEM : LBMAN_ERR_CUDA;
    return fail(st, "%s: %s", what, lbman::stats::err_string(code));
}

}  // namespace

int lbman_velocity_spectrum(lbman_solver* s, int nbins, double* E, double* counts) {
    if (!s || !E) return fail(LBMAN_ERR_ARG, "null argument");
    LB_TRY(stats_ready(s, nbins));
    s->launches += 5;  // power x3, shell binning, fold (plus cuFFT's own kernels)
    return stats_status(lbman::stats::velocity_spectrum(s->stats, s->u[s->ucur], nbins, E, counts, s->stream),
                        "velocity spectrum");
}

int lbman_q_correlation(lbman_solver* s, int nbins, double* C, double* counts, double* xi) {
    if (!s || !C) return fail(LBMAN_ERR_ARG, "null argument");
    LB_TRY(stats_ready(s, nbins));
    s->launches += 6;  // power x4, shell binning, fold (plus cuFFT's own kernels)
    LB_TRY(stats_status(lbman::stats::q_correlation(s->stats, s->q[s->qcur], nbins, C, counts, s->stream),
                        "Q correlation"));
    if (xi) {
        *xi = -1.0;
        const double target = std::exp(-1.0);
        for (int b = 1; b < nbins; ++b) {
            if (C[b] < target) {
                *xi = (b - 1) + (C[b - 1] - target) / (C[b - 1] - C[b]);
                break;
            }
        }
    }
    return LBMAN_OK;
}

int lbman_statistics(lbman_solver* s, lbman_stats* out) {
    if (!s || !out) return fail(LBMAN_ERR_ARG, "null argument");
    LB_TRY(stats_ready(s, 2));
    std::memset(out, 0, sizeof(*out));
    double m1 = 0.0, m2 = 0.0;
    s->launches += 2;
    LB_TRY(stats_status(lbman::stats::speed_moments(s->stats, s->u[s->ucur], &m1, &m2, s->stream), "speed moments"));
    out->mean_speed = m1;
    out->rms_speed = std::sqrt(m2);
    lbman_diag d;
    LB_TRY(lbman_reduce(s, LBMAN_DIAG_DEFECTS, &d));
    out->defect_faces = d.defect_faces;
    out->defect_density = d.defect_faces >= 0 ? (double)d.defect_faces / (double)s->P.V : -1.0;
    return LBMAN_OK;
}

int lbman_defect_lines(lbman_solver* s, lbman_defects* info, double* points, int64_t points_cap,
                       int64_t* line_offsets, int64_t offsets_cap) {
    if (!s || !info) return fail(LBMAN_ERR_ARG, "null argument");
    if (!s->uploaded) return fail(LBMAN_ERR_STATE, "defect lines before upload");
    if (s->slab) return fail(LBMAN_ERR_UNSUPPORTED, "defect lines of a slab: download the slabs and assemble the box");
    const int nx = s->P.nx, ny = s->P.ny, nz = s->P.nz;
    if (nx < 2 || ny < 2 || nz < 2) return fail(LBMAN_ERR_ARG, "defect lines need at least 2 cells per side");
    LB_TRY(set_device(s));
    const int64_t nf = (int64_t)nx * (ny - 1) * (nz - 1) + (int64_t)(nx - 1) * ny * (nz - 1) +
                       (int64_t)(nx - 1) * (ny - 1) * nz;
    uint8_t* dflags = nullptr;
    LB_CUDA(cudaMalloc(&dflags, (size_t)nf));
    std::vector<uint8_t> flags((size_t)nf);
    int st = check_launch(s, s->ops().defects(s->P, s->q[s->qcur], dflags, (unsigned long long*)(s->red_dev + 9), s->stream),
                          "defects");
    if (st == LBMAN_OK && (cudaMemcpyAsync(flags.data(), dflags, (size_t)nf, cudaMemcpyDeviceToHost, s->stream) != cudaSuccess ||
                           cudaStreamSynchronize(s->stream) != cudaSuccess))
        st = fail(LBMAN_ERR_CUDA, "defect flags copy failed");
    cudaFree(dflags);
    if (st != LBMAN_OK) return st;
    const int64_t nfx = (int64_t)nx * (ny - 1) * (nz - 1), nfy = (int64_t)(nx - 1) * ny * (nz - 1);
    return lbman_defect_graph(nx, ny, nz, s->P.qper, flags.data(), flags.data() + nfx, flags.data() + nfx + nfy, info,
                              points, points_cap, line_offsets, offsets_cap);
}

int lbman_get_shape(lbman_solver* s, lbman_shape* out) {
    if (!s || !out) return fail(LBMAN_ERR_ARG, "null argument");
    out->kernels = s->kernels;
    out->tile_x = s->shape.tile.tcx;
    out->tile_y = s->shape.tile.tcy;
    out->zchunk = s->shape.tile.zc;
    out->threads = s->shape.qthreads;
    out->ms_per_step = 0.0;
    out->blocks = s->ops().march_blocks(s->P, s->shape, s->kernels == LBMAN_KERNELS_FUSED);
    return LBMAN_OK;
}

static int check_shape(lbman_solver* s, const lbman_shape* sh, QTile* tile) {
    if (sh->kernels != LBMAN_KERNELS_SPLIT && sh->kernels != LBMAN_KERNELS_FUSED &&
        sh->kernels != LBMAN_KERNELS_SPLIT_PAIR)
        return fail(LBMAN_ERR_ARG, "kernels must be LBMAN_KERNELS_SPLIT, LBMAN_KERNELS_FUSED or LBMAN_KERNELS_SPLIT_PAIR");
    if (s->slab && sh->kernels == LBMAN_KERNELS_FUSED)
        return fail(LBMAN_ERR_UNSUPPORTED, "slabs step with the in-place organisations");
    QTile t{sh->tile_x, sh->tile_y, sh->zchunk};
    t.pair = sh->kernels == LBMAN_KERNELS_SPLIT_PAIR;
    if (sh->zchunk < -8) return fail(LBMAN_ERR_ARG, "zchunk must be >= -8 (<= 0: balanced schedule)");
    if (t.pair && (s->prec == LBMAN_FP64 || (s->P.nx & 3) != 0))
        return fail(LBMAN_ERR_ARG, "LBMAN_KERNELS_SPLIT_PAIR needs FP32 or FP16 precision and nx a multiple of 4");
    if (s->ops().qforce_smem(t) == 0)
        return fail(LBMAN_ERR_ARG, "tile %dx%d is not compiled for this precision%s", sh->tile_x, sh->tile_y,
                    t.pair ? " and organisation" : "");
    *tile = t;
    return LBMAN_OK;
}

// Steps with the z-marching launch sh names; the point kernels' scratch stays.
static int use_shape(lbman_solver* s, const lbman_shape* sh) {
    QTile t;
    LB_TRY(check_shape(s, sh, &t));
    s->kernels = sh->kernels;
    s->point = false;
    s->shape.tile = t;
    s->shape.qthreads = s->ops().qforce_threads(t);
    return LBMAN_OK;
}

// Does the shape name the point kernels?
static bool names_point(const lbman_solver* s, const lbman_shape* sh) {
    return s->point_able && sh->kernels == s->untuned.kernels && sh->tile_x == s->untuned.tile_x &&
           sh->tile_y == s->untuned.tile_y && sh->zchunk == s->untuned.zchunk;
}

int lbman_set_shape(lbman_solver* s, const lbman_shape* sh) {
    if (!s || !sh) return fail(LBMAN_ERR_ARG, "null argument");
    LB_TRY(use_shape(s, sh));
    LB_TRY(set_device(s));
    if (names_point(s, sh)) take_point(s);
    else drop_point(s);
    return LBMAN_OK;
}

// Average step time of the current shape over n steps after one untimed
// step, CUDA events on the solver's stream.
static int time_trial(lbman_solver* s, int n, cudaEvent_t e0, cudaEvent_t e1, double* ms_per_step) {
    LB_TRY(one_step(s, false));
    cudaEventRecord(e0, s->stream);
    for (int i = 0; i < n; ++i) LB_TRY(one_step(s, false));
    cudaEventRecord(e1, s->stream);
    if (cudaEventSynchronize(e1) != cudaSuccess) return fail(LBMAN_ERR_CUDA, "autotune trial failed");
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    *ms_per_step = ms / n;
    return LBMAN_OK;
}

int lbman_autotune(lbman_solver* s, int steps_per_trial, lbman_shape* best, int* ntrials) {
    if (!s || !best) return fail(LBMAN_ERR_ARG, "null argument");
    if (!s->uploaded) return fail(LBMAN_ERR_STATE, "autotune needs an uploaded state");
    if (steps_per_trial < 1) return fail(LBMAN_ERR_ARG, "steps_per_trial must be >= 1");
    LB_TRY(set_device(s));
    const int64_t V = s->P.V;
    // Snapshot of the state the trials will advance.
    const size_t fb = 15 * V * s->sbytes, qb = 5 * V * s->rbytes, ub = 3 * V * s->rbytes, rb = V * s->rbytes;
    char* snap = nullptr;
    LB_CUDA(cudaMalloc(&snap, fb + qb + ub + rb + ub));
    const int fc = s->fcur, qc = s->qcur, uc = s->ucur;
    const int fphase = s->fphase;
    const int64_t steps0 = s->steps;
    auto copy_state = [&](bool save) -> cudaError_t {
        void* dst[5] = {snap, snap + fb, snap + fb + qb, snap + fb + qb + ub, snap + fb + qb + ub + rb};
        void* src[5] = {s->f[fc], s->q[qc], s->u[uc], s->rho, s->F};
        const size_t n[5] = {fb, qb, ub, rb, ub};
        for (int k = 0; k < 5; ++k) {
            cudaError_t e = save ? cudaMemcpyAsync(dst[k], src[k], n[k], cudaMemcpyDeviceToDevice, s->stream)
                                 : cudaMemcpyAsync(src[k], dst[k], n[k], cudaMemcpyDeviceToDevice, s->stream);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    };
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    int status = LBMAN_OK, count = 0;
    lbman_shape orig, cur{}, win{};
    std::vector<lbman_shape> trials;
    bool point = false;
    double point_ms = 1e30;
    lbman_get_shape(s, &orig);
    win = orig;
    win.ms_per_step = 1e30;
    if (copy_state(true) != cudaSuccess || cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) {
        status = fail(LBMAN_ERR_CUDA, "autotune set-up failed");
    } else {
        point = s->point_able && use_shape(s, &s->untuned) == LBMAN_OK && take_point(s);
        if (point) {  // the point kernels: one trial, at the length of the final ones
            status = time_trial(s, 3 * steps_per_trial, e0, e1, &point_ms);
            ++count;
        }
        for (int k : {LBMAN_KERNELS_SPLIT, LBMAN_KERNELS_FUSED, LBMAN_KERNELS_SPLIT_PAIR}) {
            if (status != LBMAN_OK) break;
            if (k == LBMAN_KERNELS_SPLIT_PAIR && (s->prec == LBMAN_FP64 || (s->P.nx & 3) != 0)) continue;
            // the fused organisation needs a second population buffer; a box
            // too large for it is tuned over the in-place organisations only
            if (k == LBMAN_KERNELS_FUSED && (s->slab || ensure_f1(s) != LBMAN_OK)) continue;
            for (const auto& t : kTileList) {
                QTile q{t[0], t[1], 1};
                q.pair = k == LBMAN_KERNELS_SPLIT_PAIR;
                if (s->ops().qforce_smem(q) == 0) continue;
                // the balanced one-wave schedule, then fixed chunks around the
                // default chunk length
                const int nzo = s->P.zhi - s->P.zlo;
                const int z0 = default_zchunk(s->P.nx, s->P.ny, nzo, t[0], t[1], s->num_sms);
                // plus 32- and 64-plane chunks: many waves of medium marches keep
                // the blocks of an SM out of step (measured best for the pair
                // kernel on large boxes)
                int zs[8] = {0, -2, -3, z0, std::max(4, z0 / 2), std::min(nzo, 2 * z0), 32, 64};
                for (int zi = 0; zi < 8 && status == LBMAN_OK; ++zi) {
                    bool seen = false;
                    for (int zj = 0; zj < zi; ++zj) seen = seen || zs[zj] == zs[zi];
                    if (seen || (zi >= 6 && zs[zi] >= nzo)) continue;
                    cur = {k, t[0], t[1], zs[zi], 0, 0.0};
                    if (point && names_point(s, &cur)) continue;
                    if (use_shape(s, &cur) != LBMAN_OK) continue;
                    if ((status = time_trial(s, steps_per_trial, e0, e1, &cur.ms_per_step)) != LBMAN_OK) break;
                    ++count;
                    trials.push_back(cur);
                }
            }
        }
        // Short trials are noisy (clocks move under the power cap): the best
        // few are timed again with three times the steps and the winner is
        // taken among them.
        std::sort(trials.begin(), trials.end(),
                  [](const lbman_shape& a, const lbman_shape& b) { return a.ms_per_step < b.ms_per_step; });
        for (size_t i = 0; i < trials.size() && i < 4 && status == LBMAN_OK; ++i) {
            cur = trials[i];
            if (use_shape(s, &cur) != LBMAN_OK) continue;
            if ((status = time_trial(s, 3 * steps_per_trial, e0, e1, &cur.ms_per_step)) != LBMAN_OK) break;
            ++count;
            if (cur.ms_per_step < win.ms_per_step) win = cur;
        }
    }
    // Restore the state and the indices it lived in, then adopt the winner.
    if (copy_state(false) != cudaSuccess && status == LBMAN_OK) status = fail(LBMAN_ERR_CUDA, "state restore failed");
    cudaStreamSynchronize(s->stream);
    s->fcur = fc; s->qcur = qc; s->ucur = uc; s->fphase = fphase; s->steps = steps0;
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaFree(snap);
    if (status != LBMAN_OK) {
        lbman_set_shape(s, &orig);
        return status;
    }
    if (point && point_ms <= win.ms_per_step) {
        win = s->untuned;
        win.ms_per_step = point_ms;
    }
    lbman_set_shape(s, &win);
    lbman_get_shape(s, best);
    best->ms_per_step = win.ms_per_step;
    if (ntrials) *ntrials = count;
    return LBMAN_OK;
}

// ---- z-slabs ---------------------------------------------------------------

int lbman_create_slab(const lbman_config* cfg, int nz_global, int z_offset, lbman_solver** out) {
    if (!cfg || !out) return fail(LBMAN_ERR_ARG, "null argument");
    *out = nullptr;
    LB_TRY(validate(*cfg));
    const int nzl = cfg->nz;
    if (nzl < 2) return fail(LBMAN_ERR_ARG, "a slab owns at least 2 planes (the Q halo is 2 planes deep)");
    if (z_offset < 0 || nz_global < nzl || z_offset > nz_global - nzl)
        return fail(LBMAN_ERR_ARG, "planes [%d, %d) are not inside a box of %d planes", z_offset, z_offset + nzl, nz_global);
    for (int k = 4; k < 6; ++k)
        if (cfg->face[k].qbc != LBMAN_Q_PERIODIC || cfg->face[k].ubc != LBMAN_U_PERIODIC)
            return fail(LBMAN_ERR_UNSUPPORTED, "z-slabs need periodic z faces (Q and velocity)");
    if (cfg->kernels == LBMAN_KERNELS_FUSED)
        return fail(LBMAN_ERR_UNSUPPORTED, "slabs step with the in-place organisations (SPLIT or SPLIT_PAIR)");
    if ((double)cfg->nx * cfg->ny * (nzl + 4) >= 2147483648.0)
        return fail(LBMAN_ERR_UNSUPPORTED, "a slab with its ghost planes must hold fewer than 2^31 cells");
    lbman_config c = *cfg;
    c.nz = nzl + 4;
    lbman_solver* s = nullptr;
    LB_TRY(lbman_create(&c, &s));
    s->slab = true;
    drop_point(s);  // the point kernels cover whole boxes
    s->point_able = false;
    s->nz_global = nz_global;
    s->z_offset = z_offset;
    SimParams& P = s->P;
    P.zlo = 2;
    P.zhi = nzl + 2;
    P.c0 = 2 * P.nxy;
    P.c1 = (int64_t)(nzl + 2) * P.nxy;
    P.gbase = (int64_t)(z_offset - 2) * P.nxy;
    auto bail = [&](int code) {
        lbman_destroy(s);
        return code;
    };
    const int64_t V = P.V;
    // ghost planes start finite; the exchanges fill them before any read
    cudaError_t e = cudaMemsetAsync(s->f[0], 0, 15 * V * s->sbytes, s->stream);
    for (int b = 0; b < 2 && e == cudaSuccess; ++b) {
        e = cudaMemsetAsync(s->q[b], 0, 5 * V * s->rbytes, s->stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(s->u[b], 0, 3 * V * s->rbytes, s->stream);
    }
    if (e == cudaSuccess) e = cudaMemsetAsync(s->rho, 0, V * s->rbytes, s->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(s->F, 0, 3 * V * s->rbytes, s->stream);
    if (e == cudaSuccess) e = cudaMalloc(&s->fstage, 10 * P.nxy * s->sbytes);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&s->ev_ready, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&s->ev_done, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
    if (e != cudaSuccess) return bail(fail(LBMAN_ERR_CUDA, "slab set-up failed: %s", cudaGetErrorString(e)));
    *out = s;
    return LBMAN_OK;
}

int lbman_slab_info(lbman_solver* s, int* nz_global, int* z_offset, int* nz_local) {
    if (!s) return fail(LBMAN_ERR_ARG, "null solver");
    const int nzl = s->P.zhi - s->P.zlo;
    if (nz_global) *nz_global = s->slab ? s->nz_global : nzl;
    if (z_offset) *z_offset = s->slab ? s->z_offset : 0;
    if (nz_local) *nz_local = nzl;
    return LBMAN_OK;
}

// The slots whose direction crosses the low z face upward (e_z = +1) and the
// high face downward (e_z = -1), in increasing order.
static const int kUpSlots[5] = {5, 7, 8, 9, 10};
static const int kDownSlots[5] = {6, 11, 12, 13, 14};

int lbman_halo_plan(int nz_local, int phase, lbman_halo_span send[2][LBMAN_HALO_MAX_SPANS],
                    lbman_halo_span recv[2][LBMAN_HALO_MAX_SPANS], int* n) {
    if (!send || !recv || !n) return fail(LBMAN_ERR_ARG, "null argument");
    if (nz_local < 2) return fail(LBMAN_ERR_ARG, "a slab owns at least 2 planes");
    auto span = [](int field, int comp, int plane, int planes) { return lbman_halo_span{field, comp, plane, planes}; };
    if (phase == LBMAN_HALO_QU) {
        // owned -> ghost, 2 planes: the Q+force kernel reads Q and u up to 2
        // planes beyond the owned ones
        *n = 8;
        for (int k = 0; k < 8; ++k) {
            const int field = k < 5 ? LBMAN_FIELD_Q : LBMAN_FIELD_U, comp = k < 5 ? k : k - 5;
            send[0][k] = span(field, comp, 0, 2);
            send[1][k] = span(field, comp, nz_local - 2, 2);
            recv[0][k] = span(field, comp, -2, 2);
            recv[1][k] = span(field, comp, nz_local, 2);
        }
    } else if (phase == LBMAN_HALO_F_IN) {
        // before an odd in-place step: a boundary cell gathers f*_j of the
        // neighbour's boundary plane from slot opp(j) there, i.e. the slots
        // crossing the face towards the neighbour
        *n = 5;
        for (int k = 0; k < 5; ++k) {
            send[0][k] = span(LBMAN_FIELD_F, kUpSlots[k], 0, 1);
            recv[1][k] = span(LBMAN_FIELD_F, kUpSlots[k], nz_local, 1);
            send[1][k] = span(LBMAN_FIELD_F, kDownSlots[k], nz_local - 1, 1);
            recv[0][k] = span(LBMAN_FIELD_F, kDownSlots[k], -1, 1);
        }
    } else if (phase == LBMAN_HALO_F_OUT) {
        // after it: those slots, rewritten by this slab's boundary cells,
        // go back to the neighbour's boundary plane (via its staging area)
        *n = 5;
        for (int k = 0; k < 5; ++k) {
            send[0][k] = span(LBMAN_FIELD_F, kDownSlots[k], -1, 1);
            recv[1][k] = span(LBMAN_FIELD_FSTAGE, k, 1, 1);
            send[1][k] = span(LBMAN_FIELD_F, kUpSlots[k], nz_local, 1);
            recv[0][k] = span(LBMAN_FIELD_FSTAGE, k, 0, 1);
        }
    } else {
        return fail(LBMAN_ERR_ARG, "bad halo phase %d", phase);
    }
    return LBMAN_OK;
}

static void* span_ptr(lbman_solver* s, const lbman_halo_span& sp) {
    const SimParams& P = s->P;
    const int64_t plane = (int64_t)(P.zlo + sp.plane) * P.nxy;
    switch (sp.field) {
        case LBMAN_FIELD_Q: return vptr(s->q[s->qcur], sp.comp * P.V + plane, s->rbytes);
        case LBMAN_FIELD_U: return vptr(s->u[s->ucur], sp.comp * P.V + plane, s->rbytes);
        case LBMAN_FIELD_F: return vptr(s->f[s->fcur], sp.comp * P.V + plane, s->sbytes);
        default: return vptr(s->fstage, (int64_t)(sp.plane * 5 + sp.comp) * P.nxy, s->sbytes);
    }
}

// Does the phase move anything now: the population halos only around odd
// in-place steps.
static bool halo_active(const lbman_solver* s, int phase) {
    if (phase == LBMAN_HALO_F_IN) return s->fphase == F_SWAP;
    if (phase == LBMAN_HALO_F_OUT) return s->fout_pending;
    return true;
}

int lbman_halo_spans(lbman_solver* s, int phase, void* send[2][LBMAN_HALO_MAX_SPANS],
                     void* recv[2][LBMAN_HALO_MAX_SPANS], size_t* span_bytes, int* n) {
    if (!s || !send || !recv || !span_bytes || !n) return fail(LBMAN_ERR_ARG, "null argument");
    if (!s->slab) return fail(LBMAN_ERR_STATE, "not a slab (lbman_create_slab)");
    if (!s->uploaded) return fail(LBMAN_ERR_STATE, "exchange before upload");
    lbman_halo_span ps[2][LBMAN_HALO_MAX_SPANS], pr[2][LBMAN_HALO_MAX_SPANS];
    int cnt = 0;
    LB_TRY(lbman_halo_plan(s->P.zhi - s->P.zlo, phase, ps, pr, &cnt));
    *n = halo_active(s, phase) ? cnt : 0;
    *span_bytes = (size_t)(ps[0][0].planes * s->P.nxy) * (phase == LBMAN_HALO_QU ? s->rbytes : s->sbytes);
    for (int f = 0; f < 2; ++f)
        for (int k = 0; k < *n; ++k) {
            send[f][k] = span_ptr(s, ps[f][k]);
            recv[f][k] = span_ptr(s, pr[f][k]);
        }
    return LBMAN_OK;
}

int lbman_halo_done(lbman_solver* s, int phase) {
    if (!s) return fail(LBMAN_ERR_ARG, "null solver");
    if (!s->slab) return fail(LBMAN_ERR_STATE, "not a slab (lbman_create_slab)");
    if (phase == LBMAN_HALO_QU) {
        s->qu_fresh = true;
    } else if (phase == LBMAN_HALO_F_IN) {
        if (s->fphase == F_SWAP) s->fin_fresh = true;
    } else if (phase == LBMAN_HALO_F_OUT) {
        if (s->fout_pending) {
            LB_TRY(set_device(s));
            const int64_t nxy = s->P.nxy;
            for (int face = 0; face < 2; ++face)
                LB_TRY(check_launch(s, s->ops().halo_merge(s->P, s->f[s->fcur], vptr(s->fstage, face * 5 * nxy, s->sbytes),
                                                           face, s->stream),
                                    "halo_merge"));
            s->fout_pending = false;
        }
    } else {
        return fail(LBMAN_ERR_ARG, "bad halo phase %d", phase);
    }
    return LBMAN_OK;
}

int lbman_slab_exchange(lbman_solver* const* slabs, int nslabs, int phase) {
    if (!slabs || nslabs < 1) return fail(LBMAN_ERR_ARG, "no slabs");
    const int n = nslabs;
    struct Spans {
        void* send[2][LBMAN_HALO_MAX_SPANS];
        void* recv[2][LBMAN_HALO_MAX_SPANS];
        size_t bytes = 0;
        int n = 0;
    };
    std::vector<Spans> sp((size_t)n);
    int zsum = 0;
    for (int i = 0; i < n; ++i) {
        lbman_solver* s = slabs[i];
        if (!s || !s->slab) return fail(LBMAN_ERR_ARG, "slab %d is not a slab handle", i);
        if (s->z_offset != zsum || s->nz_global != slabs[0]->nz_global || s->P.nxy != slabs[0]->P.nxy ||
            s->prec != slabs[0]->prec)
            return fail(LBMAN_ERR_ARG, "slabs must tile the box in z order with one shape and precision");
        zsum += s->P.zhi - s->P.zlo;
        LB_TRY(lbman_halo_spans(s, phase, sp[i].send, sp[i].recv, &sp[i].bytes, &sp[i].n));
        if (sp[i].n != sp[0].n) return fail(LBMAN_ERR_STATE, "slabs are at different steps");
    }
    if (zsum != slabs[0]->nz_global) return fail(LBMAN_ERR_ARG, "the slabs cover %d of %d planes", zsum, slabs[0]->nz_global);
    if (sp[0].n > 0) {
        for (int i = 0; i < n; ++i) {
            LB_TRY(set_device(slabs[i]));
            LB_CUDA(cudaEventRecord(slabs[i]->ev_ready, slabs[i]->stream));
        }
        for (int j = 0; j < n; ++j) {
            lbman_solver* r = slabs[j];
            const int lo = (j + n - 1) % n, hi = (j + 1) % n;
            LB_TRY(set_device(r));
            for (int nb : {lo, hi}) {
                if (slabs[nb]->device != r->device) {
                    cudaError_t e = cudaDeviceEnablePeerAccess(slabs[nb]->device, 0);
                    if (e == cudaErrorPeerAccessAlreadyEnabled) cudaGetLastError();
                    else if (e != cudaSuccess) cudaGetLastError();  // copies are staged by the driver instead
                }
                LB_CUDA(cudaStreamWaitEvent(r->stream, slabs[nb]->ev_ready, 0));
            }
            // the low ghosts come from the lower slab's sends across its high
            // face, the high ghosts from the upper slab's sends across its low face
            for (int k = 0; k < sp[j].n; ++k) {
                LB_CUDA(cudaMemcpyAsync(sp[j].recv[0][k], sp[lo].send[1][k], sp[j].bytes, cudaMemcpyDefault, r->stream));
                LB_CUDA(cudaMemcpyAsync(sp[j].recv[1][k], sp[hi].send[0][k], sp[j].bytes, cudaMemcpyDefault, r->stream));
            }
            LB_CUDA(cudaEventRecord(r->ev_done, r->stream));
        }
        // a slab's next kernel may overwrite what its neighbours copy out
        for (int i = 0; i < n; ++i) {
            lbman_solver* s = slabs[i];
            LB_TRY(set_device(s));
            LB_CUDA(cudaStreamWaitEvent(s->stream, slabs[(i + n - 1) % n]->ev_done, 0));
            LB_CUDA(cudaStreamWaitEvent(s->stream, slabs[(i + 1) % n]->ev_done, 0));
        }
    }
    for (int i = 0; i < n; ++i) LB_TRY(lbman_halo_done(slabs[i], phase));
    return LBMAN_OK;
}

int lbman_steps_done(lbman_solver* s, int64_t* steps) {
    if (!s || !steps) return fail(LBMAN_ERR_ARG, "null argument");
    *steps = s->steps;
    return LBMAN_OK;
}

int lbman_launch_count(lbman_solver* s, int64_t* launches) {
    if (!s || !launches) return fail(LBMAN_ERR_ARG, "null argument");
    *launches = s->launches;
    return LBMAN_OK;
}

}  // extern "C"
