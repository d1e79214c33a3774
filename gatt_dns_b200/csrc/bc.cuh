// Boundary conditions on the device: applyBoundCond (reference
// source/Fortran/nseq.F90:327-599) and the generated disturbance calls
// (runDisturbances.F90; source/disturbances/lidDrivenMovement.F90, periodicSine.F90,
// source/Fortran/holdInlet.F90).
//
// The reference applies its lists strictly in order (Dirichlet U,V,W,E,P; Neumann
// U,V,W,E,P; corners; null second derivative U,V,W,E,P; disturbances), and later
// items read values earlier ones wrote.  The host flattens those lists into one
// program of box operations (BcOp) in that order and sorts them into levels: an op's level is
// one more than the highest level of the earlier ops it conflicts with (it reads or writes a
// field point that they write, or writes one that they read), so the ops of one level are
// independent whatever their order, and every op finds the values that the reference's order
// gives it.  The points of a level's ops form one index range spread over all threads; a
// barrier separates the levels.  Programs of up to 16 levels take one launch per level over the whole
// GPU (k_bc_level).  Deeper ones, the tangent, the recording and the adjoint run in one launch: one CTA
// per batch member (block barriers) where levels are small, else a cluster of up to 16 SMs (cluster
// barriers, release/acquire).
//
// What bounds it: the chain of levels, about a microsecond each (a barrier, then dependent
// loads that miss to L2).  The pressure Neumann items and the corners are therefore one op
// each (P = R E formed on the fly, not through a scratch field): the 128^2 lid-driven cavity
// has 3 levels instead of 15 phases of consecutive ops, the 800x300 boundary layer over a
// cavity 7 instead of 27.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include "pointwise.cuh"
#include "sweep.cuh"

namespace gatt {

enum BcOpCode {
    OP_SET = 0,        // F[var](box) = val
    OP_DIR_P = 1,      // R(box) = val/(gamma-1)/E(box)
    OP_NEU = 2,        // applyNeumann on F[var]: the face `box` from the next len nodes along step
    OP_P_LOAD = 3,     // P(box) = R*E
    OP_P_NEU = 4,      // applyNeumann on P
    OP_R_FROM_P = 5,   // R(box) = P/E
    OP_CORNER_E0 = 6,  // E(box) = 0
    OP_P_FROM_E = 7,   // P(box) = E
    OP_E_ADD_P = 8,    // E(box) += P
    OP_E_DIV = 9,      // E(box) /= aux
    OP_R0 = 10,        // R(box) = 0
    OP_R_ADD_P = 11,   // R(box) += P
    OP_R_DIV_E = 12,   // R(box) = R/E/aux
    OP_LID = 13,       // lidDrivenMovement on F[var](box), x coordinates at xoff, U0 = val
    OP_SINE = 14,      // periodicSine: F[var](box) += xs[xoff + i - i1] * sin(val * t)
    OP_HOLD = 15,      // holdInlet: aux fields (U, V, W, E, then R) of the box <-> hold + xoff
    // 3..5 and 6..12 in one op, without the scratch field (boxes one node thick along their
    // directions; the scratch form serves the others, and the adjoint)
    OP_PNEU = 16,      // R(face) = applyNeumann(R*E)/E
    OP_CORNER = 17     // adiabatic (var = 1): E = sum of its extrapolations / aux;
                       // R = sum of the extrapolations of R*E / E / aux; directions step[0..aux)
};

struct BcOp {
    int code;
    int var;        // 0..4 (U,V,W,R,E)
    int box[6];     // 1-based inclusive i1 i2 j1 j2 k1 k2 of the points the op runs over
    int len;        // extrapolation length
    int coef;       // 0 = neumannCoeffs, 1 = neumann2Coeffs
    int aux;        // divisor for corner averages
    int xoff;       // offset of the box's x coordinates (OP_LID), of its x factors (OP_SINE), of
                    // its values in the member's hold buffer (OP_HOLD)
    unsigned first, count;  // its points in its level's index range
    FastDiv fd_ni, fd_nij;  // dividers by the box's x extent and x-y extent
    long long step[3];      // element strides of the extrapolation directions, signed
    double val;
    long long tape; // adjoint tape: offset of this op's recorded base values (-1: none)
};

static_assert(sizeof(BcOp) % sizeof(long long) == 0, "ops are staged as 8-byte words");

// Levels of a program: ops lev_op[l] .. lev_op[l+1] make level l, lev_pts[l] points in all
// (lev holds lev_op[0 .. nlev], then lev_pts[0 .. nlev-1]).
struct BcProgram {
    const BcOp *ops;
    const unsigned *lev;
    int nops, nlev;
    int n1, n2;           // lengths of the two
    const double *coef1;  // neumannCoeffs
    const double *coef2;  // neumann2Coeffs
    const double *xs;     // disturbance coordinates (OP_LID) and x factors (OP_SINE)
    double gamma;
    int nx, ny, nz;
    // the time of the call: sp->t + tfac * sp->dt (the step's parameters on the device, so that
    // one captured program serves every step), or tfix when sp is null
    const StepParams *sp;
    double tfac, tfix;
    double *hold;         // holdInlet values, hstride per member
    long long hstride;
    int hold_save;        // 1: OP_HOLD keeps the fields (first call), 0: puts them back
};

__device__ __forceinline__ double bc_time(const BcProgram &pg)
{
    return pg.sp ? pg.sp->t + pg.tfac * pg.sp->dt : pg.tfix;
}

// periodicSine.F90:17-19: u + (amplitude sin(alpha (x_i - x_1))) sin(omega t), the x factor
// precomputed per point; the product and the sum rounded separately as the reference does
__device__ __forceinline__ double bc_sine(double u, double fx, double omega, double t)
{
    return __dadd_rn(u, __dmul_rn(fx, sin(omega * t)));
}

// lidDrivenMovement.F90:15-17 at x node i of an op's box
__device__ __forceinline__ double bc_lid(const BcProgram &pg, const BcOp &op, int i)
{
    const double *x = pg.xs + op.xoff;
    const double s = 2 * (x[i - op.box[0]] - x[0]) / (x[op.box[1] - op.box[0]] - x[0]) - 1;
    const double s2 = s * s, s4 = s2 * s2, s8 = s4 * s4, s16 = s8 * s8;
    const double pp = 1 - s16 * s2;
    return op.val * (pp * pp);
}

// holdInlet.F90 keeps u, v, w, e (and r with holdDensity): field of the v-th held value
__device__ __forceinline__ int bc_hold_field(int v) { return v < 3 ? v : (v == 3 ? 4 : 3); }

// Extrapolation terms whose loads are issued together (the sixth-order Neumann rows have six
// nodes); one load at a time waits for L2 once per term.
constexpr int kBcLen = 6;

// applyNeumann (nseq.F90:552-599) at one face point: u points to it, st steps into the domain;
// products and sums rounded one by one as the reference does (no fused multiply-add: chains of
// boundary items, with divisions by extrapolated E between them, amplify the difference)
__device__ __forceinline__ double bc_extrapolate(const double *u, long long st, int len, const double *c)
{
    double x[kBcLen];
#pragma unroll
    for (int m = 1; m <= kBcLen; m++) x[m - 1] = m <= len ? u[m * st] : 0.0;
    double v = __dmul_rn(c[0], x[0]);
#pragma unroll
    for (int m = 2; m <= kBcLen; m++)
        if (m <= len) v = __dadd_rn(v, __dmul_rn(c[m - 1], x[m - 1]));
    for (int m = kBcLen + 1; m <= len; m++) v = __dadd_rn(v, __dmul_rn(c[m - 1], u[m * st]));
    return v;
}
// the same of P = R*E
__device__ __forceinline__ double bc_extrapolate_p(const double *r, const double *e, long long st, int len,
                                                   const double *c)
{
    double x[kBcLen], y[kBcLen];
#pragma unroll
    for (int m = 1; m <= kBcLen; m++) {
        x[m - 1] = m <= len ? r[m * st] : 0.0;
        y[m - 1] = m <= len ? e[m * st] : 0.0;
    }
    double v = __dmul_rn(c[0], __dmul_rn(x[0], y[0]));
#pragma unroll
    for (int m = 2; m <= kBcLen; m++)
        if (m <= len) v = __dadd_rn(v, __dmul_rn(c[m - 1], __dmul_rn(x[m - 1], y[m - 1])));
    for (int m = kBcLen + 1; m <= len; m++)
        v = __dadd_rn(v, __dmul_rn(c[m - 1], __dmul_rn(r[m * st], e[m * st])));
    return v;
}

// Largest program that is staged in shared memory (ops, levels, coefficients; 48 KB, no opt-in
// needed); longer programs read them from global memory.
constexpr int kBcStagedBytes = 48 * 1024;
constexpr int kBcThreads = 512;   // threads of a boundary-program CTA
__host__ __device__ __forceinline__ size_t bc_stage_bytes(const BcProgram &pg)
{
    return (size_t)pg.nops * sizeof(BcOp) + (size_t)(pg.nlev + 1) * 8 + (size_t)(pg.n1 + pg.n2) * 8;
}

// Copy the program to shared memory (when it fits) and point pg there; every thread of the CTA
// calls it.  The host pads the level table to whole 8-byte words.
__device__ __forceinline__ void bc_stage(BcProgram &pg, long long *sh)
{
    if (bc_stage_bytes(pg) > (size_t)kBcStagedBytes) return;
    const int n = pg.nops * (int)(sizeof(BcOp) / sizeof(long long)), m = pg.nlev + 1;
    const long long *g = reinterpret_cast<const long long *>(pg.ops), *gl = reinterpret_cast<const long long *>(pg.lev);
    double *c1 = reinterpret_cast<double *>(sh + n + m), *c2 = c1 + pg.n1;
    for (int i = threadIdx.x; i < n; i += blockDim.x) sh[i] = g[i];
    for (int i = threadIdx.x; i < m; i += blockDim.x) sh[n + i] = gl[i];
    for (int i = threadIdx.x; i < pg.n1; i += blockDim.x) c1[i] = pg.coef1[i];
    for (int i = threadIdx.x; i < pg.n2; i += blockDim.x) c2[i] = pg.coef2[i];
    __syncthreads();
    pg.ops = reinterpret_cast<const BcOp *>(sh);
    pg.lev = reinterpret_cast<const unsigned *>(sh + n);
    pg.coef1 = c1;
    pg.coef2 = c2;
}

// fn(op, r, i, p) for every point of level lv, thread tid of nthr: r the point's index in the
// op's box (x fastest), i its x node, p its element offset.  op: the level's first op.
template <typename Fn>
__device__ __forceinline__ void bc_level(const BcProgram &pg, const BcOp *op, unsigned total, int tid, int nthr, Fn fn)
{
    for (unsigned q = tid; q < total; q += nthr) {
        while (q >= op->first + op->count) op++;
        const unsigned r = q - op->first;
        const unsigned kq = fdiv((int)r, op->fd_nij), rr = r - kq * op->fd_nij.d, jq = fdiv((int)rr, op->fd_ni);
        const int i = op->box[0] + (int)(rr - jq * op->fd_ni.d);
        const long long p = (long long)(i - 1) +
                            (long long)pg.nx * ((op->box[2] - 1 + (int)jq) + (long long)pg.ny * (op->box[4] - 1 + (int)kq));
        fn(*op, r, i, p);
    }
}

// Every level; sync() (a barrier over all nthr threads that orders their memory accesses) between
// levels.  REV: last level first.
template <bool REV = false, typename Sync, typename Fn>
__device__ __forceinline__ void bc_levels(const BcProgram &pg, int tid, int nthr, Sync sync, Fn fn)
{
    for (int l = 0; l < pg.nlev; l++) {
        if (l) sync();
        const int lv = REV ? pg.nlev - 1 - l : l;
        bc_level(pg, pg.ops + pg.lev[lv], pg.lev[pg.nlev + 1 + lv], tid, nthr, fn);
    }
}

// A member's state arrays: indexed by the op's variable, straight from the kernel parameters (a
// local pointer array would live in local memory).
struct BcFields {
    const StateSet &s;
    long long off;
    __device__ __forceinline__ BcFields(const StateSet &set, int b) : s(set), off(b * set.bstride) {}
    __device__ __forceinline__ double *operator[](int v) const { return s.v[v] + off; }
};

// One point of the program on one member: F the five state arrays (U,V,W,R,E), P a scratch
// field, tnow the time of the call.
__device__ __forceinline__ void bc_point(const BcProgram &pg, const BcFields &F, double *P, double *H, double tnow,
                                         const BcOp &op, unsigned r, int i, long long p)
{
    double *Rr = F[3], *Ee = F[4];
    const double *cf = op.coef ? pg.coef2 : pg.coef1;
    switch (op.code) {
    case OP_SET: F[op.var][p] = op.val; break;
    case OP_DIR_P: Rr[p] = op.val / (pg.gamma - 1.0) / Ee[p]; break;
    case OP_NEU: F[op.var][p] = bc_extrapolate(F[op.var] + p, op.step[0], op.len, cf); break;
    case OP_PNEU: Rr[p] = bc_extrapolate_p(Rr + p, Ee + p, op.step[0], op.len, cf) / Ee[p]; break;
    case OP_CORNER: {
        if (op.var) {
            double e = 0.0;
#pragma unroll
            for (int d = 0; d < 3; d++)
                if (d < op.aux) e = e + bc_extrapolate(Ee + p, op.step[d], op.len, cf);
            Ee[p] = e / (double)op.aux;
        }
        double v = 0.0;
#pragma unroll
        for (int d = 0; d < 3; d++)
            if (d < op.aux) v = v + bc_extrapolate_p(Rr + p, Ee + p, op.step[d], op.len, cf);
        Rr[p] = v / Ee[p] / (double)op.aux;
        break;
    }
    case OP_P_LOAD: P[p] = Rr[p] * Ee[p]; break;
    case OP_P_NEU: P[p] = bc_extrapolate(P + p, op.step[0], op.len, cf); break;
    case OP_R_FROM_P: Rr[p] = P[p] / Ee[p]; break;
    case OP_CORNER_E0: Ee[p] = 0.0; break;
    case OP_P_FROM_E: P[p] = Ee[p]; break;
    case OP_E_ADD_P: Ee[p] = Ee[p] + P[p]; break;
    case OP_E_DIV: Ee[p] = Ee[p] / (double)op.aux; break;
    case OP_R0: Rr[p] = 0.0; break;
    case OP_R_ADD_P: Rr[p] = Rr[p] + P[p]; break;
    case OP_R_DIV_E: Rr[p] = Rr[p] / Ee[p] / (double)op.aux; break;
    case OP_LID: F[op.var][p] = bc_lid(pg, op, i); break;
    case OP_SINE: F[op.var][p] = bc_sine(F[op.var][p], pg.xs[op.xoff + i - op.box[0]], op.val, tnow); break;
    case OP_HOLD:
        for (int v = 0; v < op.aux; v++) {
            double *h = H + op.xoff + (long long)v * op.count + r;
            if (pg.hold_save) *h = F[bc_hold_field(v)][p];
            else F[bc_hold_field(v)][p] = *h;
        }
        break;
    default: break;
    }
}

// The whole program on one member.
template <typename Sync>
__device__ __forceinline__ void bc_run(const BcProgram &pg, const BcFields &F, double *P, double *H, int tid, int nthr,
                                       Sync sync)
{
    const double tnow = bc_time(pg);
    bc_levels(pg, tid, nthr, sync,
              [&](const BcOp &op, unsigned r, int i, long long p) { bc_point(pg, F, P, H, tnow, op, r, i, p); });
}

// One level over the whole grid (blockIdx.y: member); dynamic shared memory: the level's ops.
__global__ void __launch_bounds__(256) k_bc_level(BcProgram pg, const __grid_constant__ StateSet q, double *Pbase,
                                                  long long pstride, int lv, int op0, int nops, unsigned total)
{
    extern __shared__ long long bc_sh[];
    pdl_launch();
    const long long *g = reinterpret_cast<const long long *>(pg.ops + op0);
    for (int i = threadIdx.x; i < nops * (int)(sizeof(BcOp) / sizeof(long long)); i += blockDim.x) bc_sh[i] = g[i];
    __syncthreads();
    pdl_wait();
    const int b = blockIdx.y;
    const BcFields F(q, b);
    double *P = Pbase + b * pstride, *H = pg.hold ? pg.hold + b * pg.hstride : nullptr;
    const double tnow = bc_time(pg);
    bc_level(pg, reinterpret_cast<const BcOp *>(bc_sh), total, blockIdx.x * blockDim.x + threadIdx.x,
             gridDim.x * blockDim.x,
             [&](const BcOp &op, unsigned r, int i, long long p) { bc_point(pg, F, P, H, tnow, op, r, i, p); });
}

// One CTA per batch member (block barriers); dynamic shared memory: the staged program.
__global__ void __launch_bounds__(kBcThreads) k_bc(BcProgram pg, const __grid_constant__ StateSet q, double *Pbase,
                                            long long pstride)
{
    extern __shared__ long long bc_sh[];
    const int b = blockIdx.x;
    const BcFields F(q, b);
    pdl_launch();
    bc_stage(pg, bc_sh);  // (the program does not depend on the launch before this one)
    pdl_wait();
    double *H = pg.hold ? pg.hold + b * pg.hstride : nullptr;
    bc_run(pg, F, Pbase + b * pstride, H, threadIdx.x, blockDim.x, [] { __syncthreads(); });
}

// One cluster of CTAs per batch member (cluster barriers); launched with a cluster dimension.
__global__ void __launch_bounds__(kBcThreads) k_bc_cluster(BcProgram pg, const __grid_constant__ StateSet q, double *Pbase,
                                                    long long pstride)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const int b = blockIdx.x / (int)cl.num_blocks();
    const BcFields F(q, b);
    extern __shared__ long long bc_sh[];
    pdl_launch();
    bc_stage(pg, bc_sh);  // (the program does not depend on the launch before this one)
    pdl_wait();
    double *H = pg.hold ? pg.hold + b * pg.hstride : nullptr;
    bc_run(pg, F, Pbase + b * pstride, H, (int)cl.block_rank() * blockDim.x + threadIdx.x, (int)cl.num_threads(),
           [&] { cl.sync(); });
}

// ---- tangent-linear and adjoint of the program (no counterpart in the reference) -------
//
// The program is a sequence of in-place box updates; the nonlinear ones (pressure Dirichlet,
// P = R E, R = P / E, R = R / E / aux) need the base values they saw.  The tangent runs
// base and tangent side by side; the adjoint runs the ops in reverse with those base values
// read from a tape that k_bc_rec wrote while applying the program to the base state.
// Values recorded per box point, in the box's loop order: OP_DIR_P: E; OP_P_LOAD: R, E;
// OP_R_FROM_P: P, E; OP_R_DIV_E: R, E.

__host__ __device__ __forceinline__ int bc_tape_width(int code)
{
    return code == OP_DIR_P ? 1 : (code == OP_P_LOAD || code == OP_R_FROM_P || code == OP_R_DIV_E) ? 2 : 0;
}

// The forward program (scratch form) on the base, recording the tape: member b, thread tid of
// nthr, sync() a barrier over the nthr threads.
template <typename Sync>
__device__ __forceinline__ void k_bc_rec_run(int b, int tid, int nthr, Sync sync, const BcProgram &pg, const StateSet &q,
                                             double *Pbase, long long pstride, double *tape, long long tstride)
{
    const BcFields F(q, b);
    double *P = Pbase + b * pstride;
    double *Rr = F[3], *Ee = F[4];
    double *tp = tape + b * tstride;
    double *H = pg.hold ? pg.hold + b * pg.hstride : nullptr;
    const double tnow = bc_time(pg);
    bc_levels(pg, tid, nthr, sync, [&](const BcOp &op, unsigned r, int i, long long p) {
        const double *cf = op.coef ? pg.coef2 : pg.coef1;
        double *t = tp + op.tape + (long long)bc_tape_width(op.code) * r;
        switch (op.code) {
        case OP_SET: F[op.var][p] = op.val; break;
        case OP_DIR_P: t[0] = Ee[p]; Rr[p] = op.val / (pg.gamma - 1.0) / Ee[p]; break;
        case OP_NEU: F[op.var][p] = bc_extrapolate(F[op.var] + p, op.step[0], op.len, cf); break;
        case OP_P_LOAD: t[0] = Rr[p]; t[1] = Ee[p]; P[p] = Rr[p] * Ee[p]; break;
        case OP_P_NEU: P[p] = bc_extrapolate(P + p, op.step[0], op.len, cf); break;
        case OP_R_FROM_P: t[0] = P[p]; t[1] = Ee[p]; Rr[p] = P[p] / Ee[p]; break;
        case OP_CORNER_E0: Ee[p] = 0.0; break;
        case OP_P_FROM_E: P[p] = Ee[p]; break;
        case OP_E_ADD_P: Ee[p] = Ee[p] + P[p]; break;
        case OP_E_DIV: Ee[p] = Ee[p] / (double)op.aux; break;
        case OP_R0: Rr[p] = 0.0; break;
        case OP_R_ADD_P: Rr[p] = Rr[p] + P[p]; break;
        case OP_R_DIV_E: t[0] = Rr[p]; t[1] = Ee[p]; Rr[p] = Rr[p] / Ee[p] / (double)op.aux; break;
        case OP_LID: F[op.var][p] = bc_lid(pg, op, i); break;
        case OP_SINE: F[op.var][p] = bc_sine(F[op.var][p], pg.xs[op.xoff + i - op.box[0]], op.val, tnow); break;
        case OP_HOLD:  // the fields put back (the tangent and adjoint never run a first call)
            for (int v = 0; v < op.aux; v++) F[bc_hold_field(v)][p] = H[op.xoff + (long long)v * op.count + r];
            break;
        default: break;
        }
    });
}

__global__ void __launch_bounds__(kBcThreads) k_bc_rec(BcProgram pg, const __grid_constant__ StateSet q, double *Pbase,
                                                long long pstride, double *tape, long long tstride)
{
    extern __shared__ long long bc_sh[];
    bc_stage(pg, bc_sh);
    k_bc_rec_run(blockIdx.x, threadIdx.x, blockDim.x, [] { __syncthreads(); }, pg, q, Pbase, pstride, tape, tstride);
}

__global__ void __launch_bounds__(kBcThreads) k_bc_rec_cluster(BcProgram pg, const __grid_constant__ StateSet q, double *Pbase,
                                                        long long pstride, double *tape, long long tstride)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ long long bc_sh[];
    bc_stage(pg, bc_sh);
    k_bc_rec_run(blockIdx.x / (int)cl.num_blocks(), (int)cl.block_rank() * blockDim.x + threadIdx.x,
                 (int)cl.num_threads(), [&] { cl.sync(); }, pg, q, Pbase, pstride, tape, tstride);
}

// tangent of bc_extrapolate_p's sum
__device__ __forceinline__ double bc_extrapolate_dp(const double *r, const double *e, const double *dr, const double *de,
                                                    long long st, int len, const double *c)
{
    double v = 0.0;
    for (int m = 1; m <= len; m++) v = v + c[m - 1] * (dr[m * st] * e[m * st] + r[m * st] * de[m * st]);
    return v;
}

// tangent: base q (updated as k_bc does) and tangent dq (P, dP scratch); member b, thread tid
// of nthr, sync() a barrier over the nthr threads
template <typename Sync>
__device__ __forceinline__ void k_bc_tl_run(int b, int tid, int nthr, Sync sync, const BcProgram &pg, const StateSet &q,
                                            double *Pbase, const StateSet &dq, double *dPbase, long long pstride)
{
    const BcFields F(q, b), dF(dq, b);
    double *P = Pbase + b * pstride, *dP = dPbase + b * pstride;
    double *Rr = F[3], *Ee = F[4], *dR = dF[3], *dE = dF[4];
    double *H = pg.hold ? pg.hold + b * pg.hstride : nullptr;
    const double tnow = bc_time(pg);
    bc_levels(pg, tid, nthr, sync, [&](const BcOp &op, unsigned r, int i, long long p) {
        const double *cf = op.coef ? pg.coef2 : pg.coef1;
        switch (op.code) {
        case OP_SET: F[op.var][p] = op.val; dF[op.var][p] = 0.0; break;
        case OP_DIR_P: {
            const double e = Ee[p], rn = op.val / (pg.gamma - 1.0) / e;
            dR[p] = -rn / e * dE[p];
            Rr[p] = rn;
            break;
        }
        case OP_NEU:
            F[op.var][p] = bc_extrapolate(F[op.var] + p, op.step[0], op.len, cf);
            dF[op.var][p] = bc_extrapolate(dF[op.var] + p, op.step[0], op.len, cf);
            break;
        case OP_PNEU: {
            const double e = Ee[p], pv = bc_extrapolate_p(Rr + p, Ee + p, op.step[0], op.len, cf);
            const double dp = bc_extrapolate_dp(Rr + p, Ee + p, dR + p, dE + p, op.step[0], op.len, cf);
            dR[p] = dp / e - pv * dE[p] / (e * e);
            Rr[p] = pv / e;
            break;
        }
        case OP_CORNER: {
            const double aux = (double)op.aux;
            if (op.var) {
                double e = 0.0, de = 0.0;
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    if (d >= op.aux) continue;
                    e = e + bc_extrapolate(Ee + p, op.step[d], op.len, cf);
                    de = de + bc_extrapolate(dE + p, op.step[d], op.len, cf);
                }
                Ee[p] = e / aux;
                dE[p] = de / aux;
            }
            double v = 0.0, dv = 0.0;
#pragma unroll
            for (int d = 0; d < 3; d++) {
                if (d >= op.aux) continue;
                v = v + bc_extrapolate_p(Rr + p, Ee + p, op.step[d], op.len, cf);
                dv = dv + bc_extrapolate_dp(Rr + p, Ee + p, dR + p, dE + p, op.step[d], op.len, cf);
            }
            const double e = Ee[p];
            dR[p] = dv / e / aux - v * dE[p] / (e * e) / aux;
            Rr[p] = v / e / aux;
            break;
        }
        case OP_P_LOAD: dP[p] = dR[p] * Ee[p] + Rr[p] * dE[p]; P[p] = Rr[p] * Ee[p]; break;
        case OP_P_NEU:
            P[p] = bc_extrapolate(P + p, op.step[0], op.len, cf);
            dP[p] = bc_extrapolate(dP + p, op.step[0], op.len, cf);
            break;
        case OP_R_FROM_P: {
            const double e = Ee[p], pv = P[p];
            dR[p] = dP[p] / e - pv * dE[p] / (e * e);
            Rr[p] = pv / e;
            break;
        }
        case OP_CORNER_E0: Ee[p] = 0.0; dE[p] = 0.0; break;
        case OP_P_FROM_E: P[p] = Ee[p]; dP[p] = dE[p]; break;
        case OP_E_ADD_P: Ee[p] = Ee[p] + P[p]; dE[p] = dE[p] + dP[p]; break;
        case OP_E_DIV: Ee[p] = Ee[p] / (double)op.aux; dE[p] = dE[p] / (double)op.aux; break;
        case OP_R0: Rr[p] = 0.0; dR[p] = 0.0; break;
        case OP_R_ADD_P: Rr[p] = Rr[p] + P[p]; dR[p] = dR[p] + dP[p]; break;
        case OP_R_DIV_E: {
            const double rr = Rr[p], e = Ee[p], aux = (double)op.aux;
            dR[p] = dR[p] / e / aux - rr * dE[p] / (e * e) / aux;
            Rr[p] = rr / e / aux;
            break;
        }
        case OP_LID: F[op.var][p] = bc_lid(pg, op, i); dF[op.var][p] = 0.0; break;
        // an additive forcing in time: the tangent passes through
        case OP_SINE: F[op.var][p] = bc_sine(F[op.var][p], pg.xs[op.xoff + i - op.box[0]], op.val, tnow); break;
        case OP_HOLD:  // held fields are constants
            for (int v = 0; v < op.aux; v++) {
                F[bc_hold_field(v)][p] = H[op.xoff + (long long)v * op.count + r];
                dF[bc_hold_field(v)][p] = 0.0;
            }
            break;
        default: break;
        }
    });
}

__global__ void __launch_bounds__(kBcThreads) k_bc_tl(BcProgram pg, const __grid_constant__ StateSet q, double *Pbase,
                                               const __grid_constant__ StateSet dq, double *dPbase, long long pstride)
{
    extern __shared__ long long bc_sh[];
    bc_stage(pg, bc_sh);
    k_bc_tl_run(blockIdx.x, threadIdx.x, blockDim.x, [] { __syncthreads(); }, pg, q, Pbase, dq, dPbase, pstride);
}

__global__ void __launch_bounds__(kBcThreads) k_bc_tl_cluster(BcProgram pg, const __grid_constant__ StateSet q, double *Pbase,
                                                       const __grid_constant__ StateSet dq, double *dPbase,
                                                       long long pstride)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ long long bc_sh[];
    bc_stage(pg, bc_sh);
    k_bc_tl_run(blockIdx.x / (int)cl.num_blocks(), (int)cl.block_rank() * blockDim.x + threadIdx.x, (int)cl.num_threads(),
                [&] { cl.sync(); }, pg, q, Pbase, dq, dPbase, pstride);
}

// adjoint of bc_extrapolate at a face point: g = lam[face]; lam[face] = 0; lam[face + m s] += c_{m-1} g
__device__ __forceinline__ void bc_extrapolate_adj(double *lam, long long st, int len, const double *c)
{
    const double g = *lam;
    *lam = 0.0;
    for (int m = 1; m <= len; m++) lam[m * st] += c[m - 1] * g;
}

// adjoint: lam (the five variables) and lP (the scratch's lambda, zero on entry), the scratch
// form's levels in reverse.  Its levels also keep apart ops that only read the same point: their
// adjoints both add to it.
template <typename Sync>
__device__ __forceinline__ void k_bc_adj_run(int b, int tid, int nthr, Sync sync, const BcProgram &pg, const StateSet &lam,
                                             double *lPbase, long long pstride, const double *tape, long long tstride)
{
    const BcFields L(lam, b);
    double *lP = lPbase + b * pstride;
    double *lR = L[3], *lE = L[4];
    const double *tp = tape + b * tstride;
    bc_levels<true>(pg, tid, nthr, sync, [&](const BcOp &op, unsigned r, int, long long p) {
        const double *cf = op.coef ? pg.coef2 : pg.coef1;
        const double *t = tp + op.tape + (long long)bc_tape_width(op.code) * r;
        switch (op.code) {
        case OP_SET: L[op.var][p] = 0.0; break;
        case OP_DIR_P: {
            const double e = t[0], rn = op.val / (pg.gamma - 1.0) / e;
            lE[p] += -rn / e * lR[p];
            lR[p] = 0.0;
            break;
        }
        case OP_NEU: bc_extrapolate_adj(L[op.var] + p, op.step[0], op.len, cf); break;
        case OP_P_LOAD: lR[p] += t[1] * lP[p]; lE[p] += t[0] * lP[p]; lP[p] = 0.0; break;
        case OP_P_NEU: bc_extrapolate_adj(lP + p, op.step[0], op.len, cf); break;
        case OP_R_FROM_P: {
            const double pv = t[0], e = t[1];
            lP[p] += lR[p] / e;
            lE[p] += -pv / (e * e) * lR[p];
            lR[p] = 0.0;
            break;
        }
        case OP_CORNER_E0: lE[p] = 0.0; break;
        case OP_P_FROM_E: lE[p] += lP[p]; lP[p] = 0.0; break;
        case OP_E_ADD_P: lP[p] += lE[p]; break;
        case OP_E_DIV: lE[p] = lE[p] / (double)op.aux; break;
        case OP_R0: lR[p] = 0.0; break;
        case OP_R_ADD_P: lP[p] += lR[p]; break;
        case OP_R_DIV_E: {
            const double rr = t[0], e = t[1], aux = (double)op.aux;
            lE[p] += -rr / (e * e) / aux * lR[p];
            lR[p] = lR[p] / e / aux;
            break;
        }
        case OP_LID: L[op.var][p] = 0.0; break;
        case OP_SINE: break;
        case OP_HOLD:
            for (int v = 0; v < op.aux; v++) L[bc_hold_field(v)][p] = 0.0;
            break;
        default: break;
        }
    });
}

__global__ void __launch_bounds__(kBcThreads) k_bc_adj(BcProgram pg, const __grid_constant__ StateSet lam, double *lPbase,
                                                long long pstride, const double *tape, long long tstride)
{
    extern __shared__ long long bc_sh[];
    bc_stage(pg, bc_sh);
    k_bc_adj_run(blockIdx.x, threadIdx.x, blockDim.x, [] { __syncthreads(); }, pg, lam, lPbase, pstride, tape, tstride);
}

__global__ void __launch_bounds__(kBcThreads) k_bc_adj_cluster(BcProgram pg, const __grid_constant__ StateSet lam, double *lPbase,
                                                        long long pstride, const double *tape, long long tstride)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ long long bc_sh[];
    bc_stage(pg, bc_sh);
    k_bc_adj_run(blockIdx.x / (int)cl.num_blocks(), (int)cl.block_rank() * blockDim.x + threadIdx.x, (int)cl.num_threads(),
                 [&] { cl.sync(); }, pg, lam, lPbase, pstride, tape, tstride);
}

}  // namespace gatt
