// qpoint.cuh -- the time step as two kernels that need no shared memory: the
// Q stage's point update (qpoint_kernel), and the in-place LBM step that forms
// the body force from the stored stress (lbm_aa_point_kernel).  For the boxes
// on which the z-marching kernels (qforce.cuh, qpair.cuh) leave the chip idle
// or are bound by the arithmetic of their halo points.
//
//   qpoint_kernel        the Beris-Edwards update of a cell: Q_new, the stress
//                        (FP64: Sigma and tau; FP32: the row stress Pi of
//                        qforce.cuh, grouped by the axis it is differentiated
//                        along) and the Ericksen force (in F), to global memory;
//   point_force_kernel   the rest of the force added to F (the Q stage alone);
//   lbm_aa_point_kernel  the same force formed in registers by the in-place
//                        collide-and-stream, so it never goes to memory.
//
// The arithmetic is that of the z-marching kernels, value for value (what those
// keep in shared memory is what qpoint_kernel stores): one point per thread as
// qforce.cuh, packed as qpair.cuh, each with the bits of its counterpart.
//
// A thread of qpoint_kernel walks a chunk of planes of one (x, y) column and
// keeps the centre values of three planes in registers, so a plane costs its x
// and y neighbours (first-level cache) and one new centre value per field.  No
// point is updated twice and no warp waits for another; the price is the
// stress's trip through the second-level cache, or HBM for large boxes.  The
// packed FP32 kernels (qpoint2_kernel) on planes with long walks (force_in_walk,
// qpair.cuh) finish the z terms of the force in the walk, for all but a chunk's
// first and last plane: per cell 6 stress words and 3 of force go to the LBM
// kernel instead of 9 stress words, 3 of Ericksen force and the 3 of the old
// velocity.
//
// What bounds it: launches below about 10^5 cells, registers and latency up to
// a few 10^6 (11-18 warps per SM in the update), then HBM.  256^3 packed, DRAM
// bytes per cell as counted and the time they take at the copy rate (6463 GB/s):
//   FP32 update 90 B, 298 us for 234 (11 warps per SM; 330 us without the
//     prefetch, 318 us with 4-plane walks); LBM 168 B, 449 / 490 us even / odd
//     for 436 (the odd step's x-shifted accesses are unaligned)
//   FP16 update 98 B, 309 us for 255; LBM 130 B, 348 / 397 us for 337
// FP64 (64x256x256 slit): update 179 B, 192 us for 116, the FP64 pipe 62% active;
// LBM 406 B, 266 / 305 us for 263.  Whole steps before (z-marching Q kernel, then
// LBM) and with these kernels:
//   32^3 FP64             67 ->  8 us      20x100x100 FP64    150 -> 23 us
//   67x101x131 FP32      161 ->  60 us     64^3 FP32           39 -> 16 us
//   64x256x256 slit FP32 282 -> 244 us     same, FP64         898 -> 490 us
//   256^3 slit FP32      981 -> 834 us     256^3 FP64        2865 -> 2070 us
//   256^3 FP32 / FP16    909 -> 784, 811 -> 704 us
#pragma once

#include "lbm.cuh"
#include "pdl.cuh"
#include "qforce.cuh"
#include "qpair.cuh"

namespace lbman {

constexpr int kPointThreads = 128;

// Words per cell of stored stress.
template <class R>
constexpr int point_stress_words() {
    return sizeof(R) == 4 ? 9 : 8;
}

// Which wall rules are compiled in: bit 0, 1, 2 for walls (of Q or u) on the
// x, y, z axis, bit 3 for anchoring -- a superset of what the box has, so axes
// that are periodic by construction cost nothing.
enum : int { QW_X = 1, QW_Y = 2, QW_Z = 4, QW_ANCHOR = 8 };

// Offsets to a cell's neighbours; 0 where a rule takes the cell itself.
struct Nbr {
    int xm, xp, ym, yp, zm, zp;
};
__device__ __forceinline__ Nbr wrapped_nbr(const SimParams& P, int x, int y, int z) {
    Nbr o;
    const int nxy = (int)P.nxy;
    o.xm = x == 0 ? P.nx - 1 : -1;
    o.xp = x == P.nx - 1 ? 1 - P.nx : 1;
    o.ym = y == 0 ? (P.ny - 1) * P.nx : -P.nx;
    o.yp = y == P.ny - 1 ? -(P.ny - 1) * P.nx : P.nx;
    o.zm = z == 0 ? (P.nz - 1) * nxy : -nxy;
    o.zp = z == P.nz - 1 ? -(P.nz - 1) * nxy : nxy;
    return o;
}
// the clamps of q_rule (the low tag decides for both sides of an axis), of the
// stress differences (QXoff, src/offsets.h:59-83) and of v_rule
template <int QW>
__device__ __forceinline__ Nbr clamped(const SimParams& P, int x, int y, int z, Nbr o, const bool (&m)[3],
                                       const bool (&p)[3]) {
    if ((QW & QW_X) && x == 0 && m[0]) o.xm = 0;
    if ((QW & QW_X) && x == P.nx - 1 && p[0]) o.xp = 0;
    if ((QW & QW_Y) && y == 0 && m[1]) o.ym = 0;
    if ((QW & QW_Y) && y == P.ny - 1 && p[1]) o.yp = 0;
    if ((QW & QW_Z) && z == 0 && m[2]) o.zm = 0;
    if ((QW & QW_Z) && z == P.nz - 1 && p[2]) o.zp = 0;
    return o;
}
template <int QW>
__device__ __forceinline__ Nbr q_nbr(const SimParams& P, int x, int y, int z, const Nbr& o) {
    const bool m[3] = {!P.qper[0], !P.qper[2], !P.qper[4]};
    const bool p[3] = {!P.qper[1] || m[0], !P.qper[3] || m[1], !P.qper[5] || m[2]};
    return clamped<QW>(P, x, y, z, o, m, p);
}
template <int QW>
__device__ __forceinline__ Nbr stress_nbr(const SimParams& P, int x, int y, int z, const Nbr& o) {
    const bool m[3] = {!P.qper[0], !P.qper[2], !P.qper[4]}, p[3] = {!P.qper[1], !P.qper[3], !P.qper[5]};
    return clamped<QW>(P, x, y, z, o, m, p);
}
template <int QW>
__device__ __forceinline__ Nbr u_nbr(const SimParams& P, int x, int y, int z, const Nbr& o) {
    const bool m[3] = {!P.uper[0], !P.uper[2], !P.uper[4]}, p[3] = {!P.uper[1], !P.uper[3], !P.uper[5]};
    return clamped<QW>(P, x, y, z, o, m, p);
}

// The velocity's ghosts at a wall (v_ghost): the clamped value c becomes
// 2 U_wall - c, except for the tangential components at a free-slip wall
// (K.uw is zero unless the wall moves).
struct VWall {
    bool mn, pn, mt, pt;  // low / high ghost of the normal and of the tangential components
};
__device__ __forceinline__ VWall v_wall(const SimParams& P, int ax, int a, int n) {
    VWall w;
    w.mn = !P.uper[2 * ax] && a == 0;
    w.pn = !P.uper[2 * ax] && a == n - 1;
    w.mt = w.mn && P.face[2 * ax].ubc != U_SPECULAR;
    w.pt = w.pn && P.face[2 * ax + 1].ubc != U_SPECULAR;
    return w;
}
template <class R>
__device__ __forceinline__ R v_diff(const Phys<R>& K, const VWall& w, int ax, int comp, R m, R c, R p) {
    if (comp == ax ? w.mn : w.mt) m = R(2.0) * K.uw[2 * ax][comp] - c;
    if (comp == ax ? w.pn : w.pt) p = R(2.0) * K.uw[2 * ax + 1][comp] - c;
    return p - m;
}

// Rules of a column, fixed along its walk.
struct ColumnRules {
    Nbr oq, ou;        // x and y offsets of Q and u
    VWall vx, vy;
    AxisRule qx, qy;   // anchoring ghosts (QW_ANCHOR)
};

template <class R, bool UPWIND, int QW>
__device__ __forceinline__ void point_update(const SimParams& P, const Phys<R>& K, const ColumnRules& r, int z,
                                             const R* qin, const R* uin, int c,
                                             const R (&qm)[5], const R (&qc)[5], const R (&qp)[5], const R (&um)[2],
                                             const R (&uc)[3], const R (&up)[3], R qn[5], R sg[5], R ta[3], R er[3]) {
    constexpr bool COMB = sizeof(R) == 4;
    const int V = (int)P.V;
    const bool zw = (QW & QW_Z) && (z == 0 || z == P.nz - 1);  // uniform
    AxisRule qz;
    VWall vz;
    if (zw) {
        qz = q_rule(P, 2, z, P.nz);
        vz = v_wall(P, 2, z, P.nz);
    }
    QD<R> d[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const R* a = qin + (k * V + c);
        const R cc = qc[k];
        R xm = a[r.oq.xm], xp = a[r.oq.xp], ym = a[r.oq.ym], yp = a[r.oq.yp], zm = qm[k], zp = qp[k];
        if constexpr (QW & QW_ANCHOR) {
            q_apply<R>(r.qx, K, k, cc, xm, xp);
            q_apply<R>(r.qy, K, k, cc, ym, yp);
        }
        if (zw) q_apply<R>(qz, K, k, cc, zm, zp);
        d[k] = q_derivs<R, !COMB>(xm, xp, ym, yp, zm, zp, cc);
    }
    constexpr R HS = COMB ? R(1.0) : R(0.5);
    R gr[8];
#pragma unroll
    for (int comp = 0; comp < 3; ++comp) {
        const R* a = uin + (comp * V + c);
        const R cc = uc[comp];
        const R xm = a[r.ou.xm], xp = a[r.ou.xp], ym = a[r.ou.ym], yp = a[r.ou.yp];
        gr[comp * 3 + 0] = HS * ((QW & QW_X) ? v_diff<R>(K, r.vx, 0, comp, xm, cc, xp) : xp - xm);
        gr[comp * 3 + 1] = HS * ((QW & QW_Y) ? v_diff<R>(K, r.vy, 1, comp, ym, cc, yp) : yp - ym);
        if (comp < 2) {
            R zm = um[comp], zp = up[comp];
            if (zw) {
                if (vz.mn) zm = cc;
                if (vz.pn) zp = cc;
                gr[comp * 3 + 2] = HS * v_diff<R>(K, vz, 2, comp, zm, cc, zp);
            } else {
                gr[comp * 3 + 2] = HS * (zp - zm);
            }
        }
    }
    GradU<R> g;
    g.ux_x = gr[0]; g.ux_y = gr[1]; g.ux_z = gr[2];
    g.uy_x = gr[3]; g.uy_y = gr[4]; g.uy_z = gr[5];
    g.uz_x = gr[6]; g.uz_y = gr[7];
    if constexpr (COMB)
        pointwise_q_mat<R, UPWIND>(K, qc, uc[0], uc[1], uc[2], d, g, qn, sg, ta, er);
    else
        pointwise_q<R, UPWIND>(K, qc, uc[0], uc[1], uc[2], d, g, qn, sg, ta, er);
}

// Is plane z the first or last of a chunk (zm = planes per chunk - 1, a power of
// two minus 1)?  A long walk has both z neighbours of its inner planes and
// finishes g there; for these planes the force's reader adds them from the
// stored stress.
__device__ __forceinline__ bool chunk_edge(int z, int zm, int nz) {
    return (z & zm) == 0 || (z & zm) == zm || z == nz - 1;
}

// Stores of one updated cell.
template <class R>
__device__ __forceinline__ void point_store(const Phys<R>& K, int V, int c, const R qn[5], const R sg[5], const R ta[3],
                                            const R er[3], R* __restrict__ qout, R* __restrict__ stress,
                                            R* __restrict__ F) {
#pragma unroll
    for (int k = 0; k < 5; ++k) qout[k * V + c] = qn[k];
    if constexpr (sizeof(R) == 4) {
        // row stress, grouped as in qf_compute_plane
        const R a = -K.ALPHA;
        stress[0 * V + c] = sg[0] + a * qn[0];
        stress[1 * V + c] = (sg[1] - ta[0]) + a * qn[1];
        stress[2 * V + c] = (sg[2] - ta[1]) + a * qn[2];
        stress[3 * V + c] = (sg[1] + ta[0]) + a * qn[1];
        stress[4 * V + c] = sg[3] + a * qn[3];
        stress[5 * V + c] = (sg[4] - ta[2]) + a * qn[4];
        stress[6 * V + c] = (sg[2] + ta[1]) + a * qn[2];
        stress[7 * V + c] = (sg[4] + ta[2]) + a * qn[4];
        stress[8 * V + c] = -(sg[0] + sg[3]) - a * (qn[0] + qn[3]);
    } else {
#pragma unroll
        for (int k = 0; k < 5; ++k) stress[k * V + c] = sg[k];
#pragma unroll
        for (int k = 0; k < 3; ++k) stress[(5 + k) * V + c] = ta[k];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) F[k * V + c] = er[k];
}

// Column `col` (index within the plane) of planes [z0, z1).
template <class R, bool UPWIND, int QW>
__device__ __forceinline__ void qpoint_column(const SimParams& P, int x, int y, int col, int z0, int z1, bool live,
                                              const R* qin, const R* uin,
                                              R* __restrict__ qout, R* __restrict__ stress, R* __restrict__ F) {
    const Phys<R>& K = phys_ref<R>(P);
    const int V = (int)P.V, nxy = (int)P.nxy, nz = P.nz;
    ColumnRules r;
    r.ou = r.oq = wrapped_nbr(P, x, y, 0);
    r.ou = u_nbr<QW & (QW_X | QW_Y)>(P, x, y, 0, r.ou);
    r.oq = q_nbr<QW & (QW_X | QW_Y)>(P, x, y, 0, r.oq);
    if constexpr (QW & QW_X) r.vx = v_wall(P, 0, x, P.nx);
    if constexpr (QW & QW_Y) r.vy = v_wall(P, 1, y, P.ny);
    if constexpr (QW & QW_ANCHOR) {
        r.qx = q_rule(P, 0, x, P.nx);
        r.qy = q_rule(P, 1, y, P.ny);
    }
    R qm[5], qc[5], qp[5], um[2], uc[3], up[3];
    {
        const int m = (z0 == 0 ? nz - 1 : z0 - 1) * nxy + col, c = z0 * nxy + col;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            qm[k] = qin[k * V + m];
            qc[k] = qin[k * V + c];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (k < 2) um[k] = uin[k * V + m];
            uc[k] = uin[k * V + c];
        }
    }
#pragma unroll 1
    for (int z = z0; z < z1; ++z) {
        const int c = z * nxy + col, p = (z == nz - 1 ? 0 : z + 1) * nxy + col;
#pragma unroll
        for (int k = 0; k < 5; ++k) qp[k] = qin[k * V + p];
#pragma unroll
        for (int k = 0; k < 3; ++k) up[k] = uin[k * V + p];
        R qn[5], sg[5], ta[3], er[3];
        point_update<R, UPWIND, QW>(P, K, r, z, qin, uin, c, qm, qc, qp, um, uc, up, qn, sg, ta, er);
        if (live) point_store<R>(K, V, c, qn, sg, ta, er, qout, stress, F);
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            qm[k] = qc[k];
            qc[k] = qp[k];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (k < 2) um[k] = uc[k];
            uc[k] = up[k];
        }
    }
}

// Blocks of 128 threads per SM the registers are held to.  Measured on B200
// (update kernel alone, with 4-plane walks where not said): FP32, 256^3: 3 / 4 /
// 5 / 6 blocks 449 / 455 / 404 / 410 us; FP64: 2 / 3 / 4 blocks 1030 / 797 /
// 787 us at 256^3, 246 / 197 / 351 us on the 64x256x256 slit; packed FP32,
// 16-plane walks, 256^3: 2 / 3 / 4 blocks 352 / 298 / 319 us (four spill).
template <class R>
constexpr int point_min_blocks() {
    return sizeof(R) == 4 ? 5 : 3;
}
constexpr int kPairPointMinBlocks = 3;

// Block (bx, bz): cells [128 bx, 128 bx + 128) of each plane of z chunk bz.
template <class R, bool UPWIND, int QW>
__global__ void __launch_bounds__(kPointThreads, point_min_blocks<R>())
    qpoint_kernel(const __grid_constant__ SimParams P, FastDiv dnx, int zc, const R* qin,
                  const R* uin, R* __restrict__ qout, R* __restrict__ stress, R* __restrict__ F) {
    const int n = (int)P.nxy;
    int col = blockIdx.x * kPointThreads + threadIdx.x;
    const bool live = col < n;
    if (!live) col = n - 1;
    const int y = (int)fdiv((uint32_t)col, dnx), x = col - y * P.nx;
    const int z0 = (int)blockIdx.y * zc;
    pdl_begin();
    qpoint_column<R, UPWIND, QW>(P, x, y, col, z0, min(z0 + zc, P.nz), live, qin, uin, qout, stress, F);
}

// ---- two cells per thread, packed FP32 ------------------------------------------
// The point update in the packed arithmetic of qpair.cuh (its values, bit for
// bit): a thread updates the cells x, x + 1 (x even; nx a multiple of 4), so
// every field moves as one 8-byte access except the two x neighbours outside
// the pair.  F holds g (or W) negated.
__device__ __forceinline__ F2 ldg2(const float* p) { return {*reinterpret_cast<const float2*>(p)}; }
__device__ __forceinline__ void stg2(float* p, F2 v) { *reinterpret_cast<float2*>(p) = v.v; }

// The warp's 64 cells of plane z + 2 are asked into the second-level cache two
// planes ahead, one 128-byte line of Q (5 fields) or u (3) per lane: the long
// walk's only loads that miss it (256^3: 330 -> 298 us).  Short walks and the
// one-point kernel, with more warps in flight, lose by it (64^3 step 15.9 ->
// 17.2 us, 96 boxes 1130 -> 1145 us).
__device__ __forceinline__ const float* walk_prefetch_base(const float* q, const float* u, int V, int col, int n) {
    const int lane = threadIdx.x & 31, k = lane / 2;
    const int at = min(__shfl_sync(0xffffffffu, col, 0) + 32 * (lane & 1), n - 1);
    return k < 5 ? q + ((int64_t)k * V + at) : k < 8 ? u + ((int64_t)(k - 5) * V + at) : nullptr;
}
__device__ __forceinline__ void walk_prefetch(const float* base, int64_t off) {
    if (base) asm volatile("prefetch.global.L2 [%0];" ::"l"(base + off));
}

struct PairRulesX {
    int xl, xr;           // offsets of the left neighbour of x and the right one of x + 1
    Nbr o;                // y offsets (from x)
};

// What a walk of qpoint2_column does besides the update: nothing, the prefetch, or
// the prefetch and the z terms of the force (force_in_walk).
enum : int { WALK_SHORT = 0, WALK_LONG = 1, WALK_FORCE = 2 };

template <bool UPWIND, int QW, int WALK>
__device__ __forceinline__ void qpoint2_column(const SimParams& P, int x, int y, int col, int z0, int z1, bool live,
                                               const float* qin, const float* uin,
                                               float* __restrict__ qout, float* __restrict__ stress,
                                               float* __restrict__ F) {
    constexpr bool WALKS = WALK == WALK_FORCE;
    const Phys<float>& K = phys_ref<float>(P);
    const int V = (int)P.V, nxy = (int)P.nxy, nz = P.nz, x1 = x + 1;
    const Nbr w0 = wrapped_nbr(P, x, y, 0), w1 = wrapped_nbr(P, x1, y, 0);
    constexpr int XY = QW & (QW_X | QW_Y);
    const Nbr q0 = q_nbr<XY>(P, x, y, 0, w0), q1 = q_nbr<XY>(P, x1, y, 0, w1);
    const Nbr v0 = u_nbr<XY>(P, x, y, 0, w0), v1 = u_nbr<XY>(P, x1, y, 0, w1);
    const PairRulesX rq{q0.xm, 1 + q1.xp, q0}, ru{v0.xm, 1 + v1.xp, v0};
    VWall vx0, vx1, vy;
    AxisRule qx0, qx1, qy;
    if constexpr (QW & QW_X) {
        vx0 = v_wall(P, 0, x, P.nx);
        vx1 = v_wall(P, 0, x1, P.nx);
    }
    if constexpr (QW & QW_Y) vy = v_wall(P, 1, y, P.ny);
    if constexpr (QW & QW_ANCHOR) {
        qx0 = q_rule(P, 0, x, P.nx);
        qx1 = q_rule(P, 0, x1, P.nx);
        qy = q_rule(P, 1, y, P.ny);
    }
    F2 qm[5], qc[5], um[2], uc[3];
    const float* const pf = walk_prefetch_base(qin, uin, V, col, nxy);
    F2 wz[3], pzm[3];  // negated W - Pi_z(z-1)/2 of the plane before, its Pi_z
#pragma unroll
    for (int k = 0; k < 3; ++k) wz[k] = pzm[k] = f2(0.0f);
    {
        const int m = (z0 == 0 ? nz - 1 : z0 - 1) * nxy + col, c = z0 * nxy + col;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            qm[k] = ldg2(qin + (k * V + m));
            qc[k] = ldg2(qin + (k * V + c));
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (k < 2) um[k] = ldg2(uin + (k * V + m));
            uc[k] = ldg2(uin + (k * V + c));
        }
    }
#pragma unroll 1
    for (int z = z0; z < z1; ++z) {
        const int c = z * nxy + col, p = (z == nz - 1 ? 0 : z + 1) * nxy + col;
        const bool zw = (QW & QW_Z) && (z == 0 || z == nz - 1);
        if (WALK != WALK_SHORT && z + 1 < z1 && z + 2 < nz) walk_prefetch(pf, (int64_t)(z + 2) * nxy);
        AxisRule qz;
        VWall vz;
        if (zw) {
            qz = q_rule(P, 2, z, nz);
            vz = v_wall(P, 2, z, nz);
        }
        F2 qp[5], up[3];
        QD2 d[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const float* a = qin + (k * V + c);
            qp[k] = ldg2(qin + (k * V + p));
            const F2 cc = qc[k];
            float l = a[rq.xl], r = a[rq.xr];
            F2 ym = ldg2(a + rq.o.ym), yp = ldg2(a + rq.o.yp), zm = qm[k], zp = qp[k];
            if constexpr (QW & QW_ANCHOR) {
                float t = 0.0f;  // the neighbour inside the pair is never a ghost
                q_apply<float>(qx0, K, k, cc.v.x, l, t);
                q_apply<float>(qx1, K, k, cc.v.y, t, r);
                q_apply2(qy, qy, K, k, cc, ym, yp);
            }
            if (zw) q_apply2(qz, qz, K, k, cc, zm, zp);
            // x neighbours of the pair: (l, c.x+1) and (c.x, r)
            d[k].dx = f2(__fsub_rn(cc.v.y, l), __fsub_rn(r, cc.v.x));
            const F2 sx = f2(__fadd_rn(l, cc.v.y), __fadd_rn(cc.v.x, r));
            d[k].dy = yp - ym;
            d[k].dz = zp - zm;
            const F2 sy = ym + yp, sz = zm + zp;
            d[k].lap = fma2(f2(-6.0f), cc, (sx + sy) + sz);
            if (UPWIND) {
                d[k].d2x = fma2(f2(-2.0f), cc, sx);
                d[k].d2y = fma2(f2(-2.0f), cc, sy);
                d[k].d2z = fma2(f2(-2.0f), cc, sz);
            }
        }
        F2 gr[8];
#pragma unroll
        for (int comp = 0; comp < 3; ++comp) {
            const float* a = uin + (comp * V + c);
            up[comp] = ldg2(uin + (comp * V + p));
            const F2 cc = uc[comp];
            const float l = a[ru.xl], r = a[ru.xr];
            const F2 ym = ldg2(a + ru.o.ym), yp = ldg2(a + ru.o.yp);
            if constexpr (QW & QW_X)
                gr[comp * 3] = f2(v_diff<float>(K, vx0, 0, comp, l, cc.v.x, cc.v.y), v_diff<float>(K, vx1, 0, comp, cc.v.x, cc.v.y, r));
            else
                gr[comp * 3] = f2(__fsub_rn(cc.v.y, l), __fsub_rn(r, cc.v.x));
            if constexpr (QW & QW_Y)
                gr[comp * 3 + 1] = f2(v_diff<float>(K, vy, 1, comp, ym.v.x, cc.v.x, yp.v.x),
                                      v_diff<float>(K, vy, 1, comp, ym.v.y, cc.v.y, yp.v.y));
            else
                gr[comp * 3 + 1] = yp - ym;
            if (comp < 2) {
                F2 zm = um[comp], zp = up[comp];
                if (zw) {
                    if (vz.mn) zm = cc;
                    if (vz.pn) zp = cc;
                    gr[comp * 3 + 2] = f2(v_diff<float>(K, vz, 2, comp, zm.v.x, cc.v.x, zp.v.x),
                                          v_diff<float>(K, vz, 2, comp, zm.v.y, cc.v.y, zp.v.y));
                } else {
                    gr[comp * 3 + 2] = zp - zm;
                }
            }
        }
        GradU2 g;
        g.ux_x = gr[0]; g.ux_y = gr[1]; g.ux_z = gr[2];
        g.uy_x = gr[3]; g.uy_y = gr[4]; g.uy_z = gr[5];
        g.uz_x = gr[6]; g.uz_y = gr[7];
        F2 qn[5], pxy[6], pz[3], wn[3];
        pointwise_q_pair<UPWIND>(K, qc, uc[0], uc[1], uc[2], d, g, qn, pxy, pz, wn);
        if (WALKS) {
#pragma unroll
            for (int k = 0; k < 3; ++k) wn[k] = fma2(f2(K.MU), uc[k], wn[k]);
            if constexpr (QW & QW_ANCHOR) {
                AxisRule qzr = q_rule(P, 2, z, nz);
                qp_anchor_force(K, true, true, z == 0 || z == nz - 1, qx0, qx1, qy, qzr, qn, wn);
            }
        }
        if (live) {
#pragma unroll
            for (int k = 0; k < 5; ++k) stg2(qout + (k * V + c), qn[k]);
#pragma unroll
            for (int k = 0; k < 6; ++k) stg2(stress + (k * V + c), pxy[k]);
            if (!WALKS || z <= z0 + 1 || z >= z1 - 2) {
#pragma unroll
                for (int k = 0; k < 3; ++k) stg2(stress + ((6 + k) * V + c), pz[k]);
            }
            if (WALKS && z > z0 + 1) {
#pragma unroll
                for (int k = 0; k < 3; ++k) stg2(F + (k * V + c - nxy), fma2(f2(-0.5f), pz[k], wz[k]));
            }
            if (!WALKS || z == z0 || z == z1 - 1) {
#pragma unroll
                for (int k = 0; k < 3; ++k) stg2(F + (k * V + c), wn[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            wz[k] = fma2(f2(0.5f), pzm[k], wn[k]);
            pzm[k] = pz[k];
        }
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            qm[k] = qc[k];
            qc[k] = qp[k];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (k < 2) um[k] = uc[k];
            uc[k] = up[k];
        }
    }
}

// Block (bx, bz): cells [256 bx, 256 bx + 256) of each plane of z chunk bz.
template <bool UPWIND, int QW, int WALK>
__global__ void __launch_bounds__(kPointThreads, kPairPointMinBlocks)
    qpoint2_kernel(const __grid_constant__ SimParams P, FastDiv dnx, int zc, const float* qin,
                   const float* uin, float* __restrict__ qout, float* __restrict__ stress,
                   float* __restrict__ F) {
    const int n = (int)P.nxy;
    int col = 2 * (blockIdx.x * kPointThreads + threadIdx.x);
    const bool live = col < n;
    if (!live) col = n - 2;
    const int y = (int)fdiv((uint32_t)col, dnx), x = col - y * P.nx;
    const int z0 = (int)blockIdx.y * zc;
    pdl_begin();
    qpoint2_column<UPWIND, QW, WALK>(P, x, y, col, z0, min(z0 + zc, P.nz), live, qin, uin, qout, stress, F);
}

// ---- body force from the stored stress -----------------------------------------
// Force source of aa_even_cell / aa_odd_cell: the Ericksen force in F plus the
// stress divergence, the active term and -MU u.  u is read before the LBM
// step overwrites it (own cell only); stress and Q are not written by it.
// PAIR: the packed kernels' order of operations (qp_partial_force); WALKS: that of
// planes with long walks, where F holds g negated, or W in the planes next to a
// chunk boundary (zm), and only the x and y differences remain.
template <class R, int QW, bool PAIR = false, bool WALKS = false>
struct PointForce {
    static constexpr bool kNeedsPos = true;
    const SimParams& P;
    int zm;
    const R* qn;
    const R* stress;
    const R* u;
    const R* F;
    __device__ __forceinline__ void operator()(int c, const CellPos& q, R out[3]) const {
        const Phys<R>& K = phys_ref<R>(P);
        const int V = (int)P.V;
        const Nbr w = wrapped_nbr(P, q.x, q.y, q.z);
        const Nbr s = stress_nbr<QW>(P, q.x, q.y, q.z, w);
        if constexpr (WALKS) {
#pragma unroll
            for (int a = 0; a < 3; ++a) out[a] = -F[a * V + c];
            R xy[3][4];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const R* px = stress + (a * V + c);
                const R* py = stress + ((3 + a) * V + c);
                xy[a][0] = px[s.xm]; xy[a][1] = px[s.xp];
                xy[a][2] = py[s.ym]; xy[a][3] = py[s.yp];
            }
            if (chunk_edge(q.z, zm, P.nz)) {
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const R* pz = stress + ((6 + a) * V + c);
                    out[a] = force_z<R>(out[a], pz[s.zm], pz[s.zp]);
                }
            }
#pragma unroll
            for (int a = 0; a < 3; ++a) out[a] = force_xy<R>(out[a], xy[a][0], xy[a][1], xy[a][2], xy[a][3]);
            return;
        }
        const R u0[3] = {u[c], u[V + c], u[2 * V + c]};
        const R er[3] = {F[c], F[V + c], F[2 * V + c]};
        AxisRule qx, qy, qz;
        if constexpr (QW & QW_ANCHOR) {
            qx = q_rule(P, 0, q.x, P.nx);
            qy = q_rule(P, 1, q.y, P.ny);
            qz = q_rule(P, 2, q.z, P.nz);
        }
        if constexpr (PAIR) {
            const bool zpc = (QW & QW_Z) && q.z == P.nz - 1 && !P.qper[5];  // the +z neighbour is the clamp
            R f[3], zpv[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const R* px = stress + (a * V + c);
                const R* py = stress + ((3 + a) * V + c);
                const R* pz = stress + ((6 + a) * V + c);
                const R xm = px[s.xm], xp = px[s.xp], ym = py[s.ym], yp = py[s.yp], zm = pz[s.zm];
                zpv[a] = pz[s.zp];
                R t = __fsub_rn(__fadd_rn(__fsub_rn(xp, xm), __fsub_rn(yp, ym)), zm);
                if (zpc) t = __fadd_rn(t, zpv[a]);
                f[a] = __fmul_rn(t, 0.5f);
            }
            if constexpr (QW & QW_ANCHOR) {
                const R nA = -K.ALPHA, A = K.ALPHA;
                auto add = [&](int a, R k, R v) { f[a] = __fadd_rn(f[a], __fmul_rn(k, v)); };
                if (qx.m_ghost || qx.p_ghost) {
                    add(0, nA, anchor_delta<R>(qx, K, 0, qn[c]));
                    add(1, nA, anchor_delta<R>(qx, K, 1, qn[V + c]));
                    add(2, nA, anchor_delta<R>(qx, K, 2, qn[2 * V + c]));
                }
                if (qy.m_ghost || qy.p_ghost) {
                    add(0, nA, anchor_delta<R>(qy, K, 1, qn[V + c]));
                    add(1, nA, anchor_delta<R>(qy, K, 3, qn[3 * V + c]));
                    add(2, nA, anchor_delta<R>(qy, K, 4, qn[4 * V + c]));
                }
                if (qz.m_ghost || qz.p_ghost) {
                    add(0, nA, anchor_delta<R>(qz, K, 2, qn[2 * V + c]));
                    add(1, nA, anchor_delta<R>(qz, K, 4, qn[4 * V + c]));
                    add(2, A, anchor_delta<R>(qz, K, 0, qn[c]) + anchor_delta<R>(qz, K, 3, qn[3 * V + c]));
                }
            }
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                out[a] = __fsub_rn(__fmaf_rn(-K.MU, u0[a], f[a]), er[a]);
                if (!zpc) out[a] = __fmaf_rn(0.5f, zpv[a], out[a]);
            }
        } else if constexpr (sizeof(R) == 4) {
            R f[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const R* px = stress + (a * V + c);
                const R* py = stress + ((3 + a) * V + c);
                const R* pz = stress + ((6 + a) * V + c);
                const R xm = px[s.xm], xp = px[s.xp], ym = py[s.ym], yp = py[s.yp], zm = pz[s.zm], zp = pz[s.zp];
                f[a] = R(0.5) * (xp - xm) + R(0.5) * (yp - ym) + R(0.5) * (zp - zm);
            }
            if constexpr (QW & QW_ANCHOR) {
                // anchoring walls: the Q_new ghost differs from the clamp (anchor_delta)
                if (qx.m_ghost || qx.p_ghost) {
                    f[0] += -K.ALPHA * anchor_delta<R>(qx, K, 0, qn[c]);
                    f[1] += -K.ALPHA * anchor_delta<R>(qx, K, 1, qn[V + c]);
                    f[2] += -K.ALPHA * anchor_delta<R>(qx, K, 2, qn[2 * V + c]);
                }
                if (qy.m_ghost || qy.p_ghost) {
                    f[0] += -K.ALPHA * anchor_delta<R>(qy, K, 1, qn[V + c]);
                    f[1] += -K.ALPHA * anchor_delta<R>(qy, K, 3, qn[3 * V + c]);
                    f[2] += -K.ALPHA * anchor_delta<R>(qy, K, 4, qn[4 * V + c]);
                }
                if (qz.m_ghost || qz.p_ghost) {
                    f[0] += -K.ALPHA * anchor_delta<R>(qz, K, 2, qn[2 * V + c]);
                    f[1] += -K.ALPHA * anchor_delta<R>(qz, K, 4, qn[4 * V + c]);
                    f[2] += K.ALPHA * (anchor_delta<R>(qz, K, 0, qn[c]) + anchor_delta<R>(qz, K, 3, qn[3 * V + c]));
                }
            }
#pragma unroll
            for (int a = 0; a < 3; ++a) out[a] = er[a] + (f[a] - K.MU * u0[a]);
        } else {
            // differences of Q_new (wall ghosts), Sigma and tau (index clamp);
            // those active_passive_force does not use are never formed
            const Nbr o = q_nbr<QW>(P, q.x, q.y, q.z, w);
            R dQ[5][3], dS[3][5], dT[3][3];
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                const R* a = qn + (k * V + c);
                R xm = a[o.xm], xp = a[o.xp], ym = a[o.ym], yp = a[o.yp], zm = a[o.zm], zp = a[o.zp];
                if constexpr (QW & QW_ANCHOR) {
                    const R cc = a[0];
                    q_apply<R>(qx, K, k, cc, xm, xp);
                    q_apply<R>(qy, K, k, cc, ym, yp);
                    q_apply<R>(qz, K, k, cc, zm, zp);
                }
                dQ[k][0] = R(0.5) * (xp - xm);
                dQ[k][1] = R(0.5) * (yp - ym);
                dQ[k][2] = R(0.5) * (zp - zm);
            }
#pragma unroll
            for (int v = 0; v < 8; ++v) {
                const R* a = stress + (v * V + c);
                const R ddx = R(0.5) * (a[s.xp] - a[s.xm]), ddy = R(0.5) * (a[s.yp] - a[s.ym]);
                const R ddz = R(0.5) * (a[s.zp] - a[s.zm]);
                if (v < 5) { dS[0][v] = ddx; dS[1][v] = ddy; dS[2][v] = ddz; }
                else { dT[0][v - 5] = ddx; dT[1][v - 5] = ddy; dT[2][v - 5] = ddz; }
            }
            active_passive_force<R>(K, dQ, dS, dT, u0[0], u0[1], u0[2], er, out);
        }
    }
};

template <class R, int QW, bool PAIR = false, bool WALKS = false>
__global__ void __launch_bounds__(256)
    point_force_kernel(const __grid_constant__ SimParams P, FastDiv dnx, FastDiv dnxy, int zm, const R* qn,
                       const R* stress, const R* u, R* F) {
    const int c = (int)(blockIdx.x * 256 + threadIdx.x);
    pdl_begin();
    if (c >= (int)P.V) return;
    const int V = (int)P.V;
    R out[3];
    PointForce<R, QW, PAIR, WALKS>{P, zm, qn, stress, u, F}(c, cell_pos<int>(P, c, dnx, dnxy), out);
#pragma unroll
    for (int k = 0; k < 3; ++k) F[k * V + c] = out[k];
}

// PointForce, also stored to F when last (the body force a caller may download).
template <class R, int QW, bool PAIR, bool WALKS = false>
struct KeptPointForce {
    static constexpr bool kNeedsPos = true;
    PointForce<R, QW, PAIR, WALKS> pf;
    R* F;
    int last;
    __device__ __forceinline__ void operator()(int c, const CellPos& q, R out[3]) const {
        pf(c, q, out);
        if (last) {
            const int V = (int)pf.P.V;
#pragma unroll
            for (int k = 0; k < 3; ++k) F[k * V + c] = out[k];
        }
    }
};

// The packed force of the cells c, c + 1 (c even) of a box without walls, for
// aa_even_h2 / aa_odd_h2: the pair's own values and its y and z neighbours as
// 8-byte accesses, the x differences from four consecutive cells.
struct PairPointForce {
    const SimParams& P;
    const float* stress;
    const float* u;
    float* F;
    int last;
    struct Values {
        float v[2][3];
        template <int I>
        __device__ __forceinline__ void get(float f[3]) const {
#pragma unroll
            for (int a = 0; a < 3; ++a) f[a] = v[I][a];
        }
    };
    __device__ __forceinline__ static float2 ld(const float* p) { return *reinterpret_cast<const float2*>(p); }
    __device__ __forceinline__ static float sum(float xm, float xp, float ym, float yp, float zm, float zp, float nmu,
                                                float u, float er) {
        const float f = __fmul_rn(__fsub_rn(__fadd_rn(__fsub_rn(xp, xm), __fsub_rn(yp, ym)), zm), 0.5f);
        return __fmaf_rn(0.5f, zp, __fsub_rn(__fmaf_rn(nmu, u, f), er));
    }
    __device__ __forceinline__ Values begin(int c, const CellPos& q) const {
        const int V = (int)P.V;
        const float nmu = -phys_ref<float>(P).MU;
        const Nbr w = wrapped_nbr(P, q.x, q.y, q.z);
        const int xr = q.x + 2 == P.nx ? 2 - P.nx : 2;
        Values o;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float* sx = stress + (a * V + c);
            const float* sy = stress + ((3 + a) * V + c);
            const float* sz = stress + ((6 + a) * V + c);
            const float2 px = ld(sx), ym = ld(sy + w.ym), yp = ld(sy + w.yp), zm = ld(sz + w.zm), zp = ld(sz + w.zp);
            const float2 ua = ld(u + (a * V + c)), er = ld(F + (a * V + c));
            const float l = sx[w.xm], r = sx[xr];
            o.v[0][a] = sum(l, px.y, ym.x, yp.x, zm.x, zp.x, nmu, ua.x, er.x);
            o.v[1][a] = sum(px.x, r, ym.y, yp.y, zm.y, zp.y, nmu, ua.y, er.y);
        }
        if (last) {
#pragma unroll
            for (int a = 0; a < 3; ++a)
                *reinterpret_cast<float2*>(F + (a * V + c)) = make_float2(o.v[0][a], o.v[1][a]);
        }
        return o;
    }
};

// In-place LBM step with the force formed on the fly.  last: rho and the body
// force are also written everywhere, as after the last step of a call.
template <class R, class S, bool DEV, int WM, int QW, bool ODD, bool PAIR = false, bool WALKS = false>
__global__ void __launch_bounds__(kPointThreads)
    lbm_aa_point_kernel(const __grid_constant__ SimParams P, FastDiv dnx, FastDiv dnxy, int zm, S* f,
                        const R* qn, const R* stress, R* F, R* __restrict__ rho_buf, R* u, int last) {
    const int c = (int)(blockIdx.x * kPointThreads + threadIdx.x);
    pdl_begin();
    if (c >= (int)P.V) return;
    const KeptPointForce<R, QW, PAIR, WALKS> force{{P, zm, qn, stress, u, F}, F, last};
    if constexpr (ODD) aa_odd_cell<R, S, DEV, WM, int>(P, dnx, dnxy, c, f, force, rho_buf, u, last);
    else aa_even_cell<R, S, DEV, WM, int>(P, dnx, dnxy, c, f, force, rho_buf, u, last);
}

// The same for FP16 storage without walls and an even nx, packed arithmetic:
// two cells per thread (aa_even_h2, aa_odd_h2), because 2-byte accesses of one
// cell leave the load-store path, not HBM, as the bound.  Whole 256^3 step: one
// cell 760 us, two cells 703 us.
template <bool DEV, bool ODD>
__global__ void __launch_bounds__(256, 3)
    lbm_aa_point_h2_kernel(const __grid_constant__ SimParams P, FastDiv dnx, FastDiv dnxy, __half* f,
                           const float* stress, float* F, float* __restrict__ rho_buf, float* u, int last) {
    const int c = 2 * (int)(blockIdx.x * 256 + threadIdx.x);
    pdl_begin();
    if (c >= (int)P.V) return;
    const PairPointForce force{P, stress, u, F, last};
    const CellPos q = cell_pos<int>(P, c, dnx, dnxy);
    if constexpr (ODD) aa_odd_h2<DEV, int>(P, c, q, f, force, rho_buf, u, last);
    else aa_even_h2<DEV, int>(P, c, q, f, force, rho_buf, u, last);
}

}  // namespace lbman
