// Compact line solves of any length for sm_100a: the form of solveSystem{X,Y,Z}[per] (reference
// source/Fortran/derivs.F90:556-948) for lines that the tensor-copy solver (rsweep.cuh) does not
// take -- odd or ragged lengths, odd grids, several long matrix types -- and for launches too
// small to fill the GPU with its 32-line tiles.
//
// Same recurrences and block recombination as rsweep.cuh.  A thread keeps 16 rows of one line in
// registers (plus NR-1 halo rows either side).  A warp holds LL lines times 32/LL row blocks, a
// tile the ceil(N/16) blocks of LL lines; rows past the line's end are identity rows (host
// records).  Narrow tiles (a warp holds four blocks or more) join the blocks in two steps, four to
// a group by shuffles inside the warp and then group to group through shared memory; wide ones
// block to block through shared memory, or (GROUPS) in the narrow ones' order, so that the x+y
// sweep of a batch can take wide tiles and keep the bits of a member alone.
//
// Persistent CTAs walk the tiles.  A tile is staged in shared memory by 8-byte asynchronous
// copies, which need no alignment beyond the element's and so take every grid: x lines
// [line][row] with one pad per 16 rows and a line pitch of 4 (mod 16) words for 4 lines, 2 for 8,
// odd for 16 and 32; y/z rows [row][line] with LL pads per 16 rows for 4 or 8 lines.  Both make the
// 16-row-strided register loads conflict-free.  With two stages the next tile streams in during
// the solve.
//
// The coefficients are staged too: records of six doubles a row of the type of the tile's first
// line (kept while it stays the same; a tile's lines of other types read theirs from global
// memory: staging every type left one CTA an SM on the 400-point x lines of a plate boundary
// layer), and the band rows of the blocks that are not uniform (a compact scheme's band is the same on all rows but those
// near walls and inside buffer zones; the uniform band is a launch constant).  Read through L1
// instead, with the first CTA of every SM waiting for L2 row by row, an x sweep of four fields
// of the 128^2 grid took 7 us against 4.5 for the tensor-copy solver.
#pragma once

#include "sweep.cuh"

namespace gatt {

constexpr int kLineRows = 16;  // rows a thread holds
constexpr int kLineQ = 6;      // doubles of a compact row record: (fA, fB), (bC, pi), (D, rho)

// Threads a CTA may have, the launch bound of an instantiation: 512 for bands of 6 and 7 (128
// registers a thread), else 768 for tiles of 32 lines (80 registers) and 640 for narrower ones, whose
// CTAs are small (96).  Spills (bytes stored / loaded, -Xptxas -v): bands of 2 and 3 at most 80/44;
// band 4, that of the walled fourth-order schemes, the most: 16/16 to 104/100 in tiles of up to 16
// lines, 116/112 in the x+y sweep of walled lines (156/156 at most), 136/116 to 228/136 with 32 lines
// and 376/260 to 440/312 in the x+y sweep of 32; band 5 at most 52/52, 212/148 in that sweep.
__host__ __device__ constexpr int line_bound(int nR, int LL) { return nR >= 6 ? 512 : LL == 32 ? 768 : 640; }
// Longest line: 96 blocks, 64 for bands of 6 and 7; over 80 blocks tiles of 4 lines only.
__host__ __device__ constexpr int line_max_rows(int nR) { return nR >= 6 ? 1024 : 1536; }

// Pitch of an x line in shared memory (doubles).
__host__ __device__ __forceinline__ int line_pitch(int N, int LL)
{
    const int need = N + (N >> 4);
    if (LL >= 16) return need | 1;
    const int odd = 16 / LL;  // 2 (8 lines) or 4 (4 lines) words, mod 16
    return (need - odd + 15) / 16 * 16 + odd;
}

// Doubles of one staged tile.
__host__ __device__ __forceinline__ int line_tile_doubles(bool xd, int N, int LL)
{
    const int n = xd ? LL * line_pitch(N, LL) : N * LL + (LL <= 8 ? (N + 15) / 16 * LL : 0);
    return (n + 1) & ~1;
}

// Doubles of one type's records: P blocks of 16 rows, two pads after each (blocks of one warp
// then sit in different banks), and the corner couplings (cA, cC).
__host__ __device__ __forceinline__ int line_type_doubles(int P) { return P * (kLineRows * kLineQ + 2) + 2; }
// Doubles of one block of non-uniform band rows.
__host__ __device__ __forceinline__ int line_band_doubles(int Wp) { return kLineRows * Wp + 2; }

// Values of a line in an exchange region: its groups of four blocks (narrow tiles) or its blocks.
__host__ __device__ __forceinline__ int line_slots(int P, int LL) { return LL <= 8 ? (P + 3) / 4 : P; }

// Coefficients of a k_lsweep launch (SweepArgs holds the rest).
struct LineArgs {
    const double *Q;   // [type][line_type_doubles]
    const double *S;   // [nspecial][line_band_doubles]
    const int *blk;    // [type][P]: -1 (uniform band) or the block's index in S
    int nspecial;
    int stageS;          // S is copied to shared memory
    double band[16];     // the uniform band
    FastDiv fd_ntiles, fd_nf;
};

__host__ __device__ __forceinline__ size_t line_smem_bytes(bool xd, int N, int P, int LL, int nst, int nspecial,
                                                           int Wp, bool stageS)
{
    size_t n = (size_t)nst * line_tile_doubles(xd, N, LL) + 5 * (size_t)line_slots(P, LL) * LL + line_type_doubles(P);
    if (stageS) n += (size_t)nspecial * line_band_doubles(Wp);
    return n * sizeof(double);
}

__device__ __forceinline__ void cp_async8(double *dst, const double *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One direction's tiles job0, job0 + jstep, ...  a.Nreal: rows of a line, a.P: blocks, a.nst:
// stages (1 or 2), a.tiles_per_row: y/z tiles of LL points per row of x, a.njobs: tiles x fields
// x members.  The CTA's first ceil(P LL / 32) warps run it, the others leave.
template <bool XD, bool PER, int NR, int LL, bool GROUPS>
__device__ __forceinline__ void line_run(const SweepArgs &a, const LineArgs &c, int job0, int jstep)
{
    constexpr int H = NR - 1, W = 2 * NR - 1, WP = (W + 3) / 4 * 4, M = kLineRows, Q6 = kLineQ;
    constexpr int BB = 32 / LL;         // row blocks in a warp
    constexpr int YP = LL <= 8 ? LL : 0;  // pads per 16 rows of a y/z tile
    extern __shared__ __align__(16) double lsm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (a.P * LL + 31) >> 5;
    const int T = nw * 32;
    if (warp >= nw) return;
    auto sync = [&] { asm volatile("bar.sync 1, %0;" ::"r"(T) : "memory"); };
    const int l = lane & (LL - 1), sub = lane / LL;
    const int p = warp * BB + sub, sp = p * M;
    const int N = a.Nreal, P = a.P;
    constexpr bool narrow = LL <= 8;     // a warp holds whole groups of four blocks
    const int NS = line_slots(P, LL), sg = sub & 3, gi = narrow ? warp * (BB / 4) + (sub >> 2) : p >> 2;
    const int ng = (P + 3) / 4;
    const int pitch = XD ? line_pitch(N, LL) : 0, tsize = line_tile_doubles(XD, N, LL);
    const int td = line_type_doubles(P), bd = line_band_doubles(WP);

    // coefficients: one type's records and (where they fit) the band rows
    double *sx = lsm + a.nst * tsize, *sc = sx + 5 * NS * LL;
    auto stage_type = [&](int t0) {
        for (int i = threadIdx.x; i < td; i += T) cp_async8(sc + i, c.Q + t0 * td + i);
    };
    const double *S = c.S;
    if (c.stageS) {
        for (int i = threadIdx.x; i < c.nspecial * bd; i += T) cp_async8(sc + td + i, c.S + i);
        S = sc + td;
    }
    double *xs = sx + l;

    // a job's first line, its lines, and the first line's offset in the field sets
    struct Tile {
        int L0, nl, f, b;
        long long base;
    };
    auto tile_of = [&](int job) {
        const int fb = fdiv(job, c.fd_ntiles), tile = job - fb * a.ntiles;
        Tile q;
        q.b = fdiv(fb, c.fd_nf);
        q.f = fb - q.b * a.nf;
        if (XD) {
            q.L0 = tile * LL;
            q.nl = min(LL, a.nlines - q.L0);
            q.base = (long long)q.L0 * N;
        } else {
            const int o = fdiv(tile, a.fd_tpr), i0 = (tile - o * a.tiles_per_row) * LL;
            q.L0 = i0 + a.nx * o;
            q.nl = min(LL, a.nx - i0);
            q.base = i0 + (long long)o * a.os;
        }
        return q;
    };
    // x lines: warp w copies lines w, w + nw, ...; rows lane + 32 k sit 34 words apart
    auto issue = [&](const Tile &q, double *dst) {
        const double *in = a.in + (long long)q.b * a.in_bstride + (long long)a.in_slot[q.f] * a.npts + q.base;
        if (XD) {
            for (int n = warp; n < q.nl; n += nw) {
                const double *src = in + (long long)n * N + lane;
                double *d = dst + n * pitch + lane + (lane >> 4);
#pragma unroll 4
                for (int r = lane; r < N; r += 32, src += 32, d += 34) cp_async8(d, src);
            }
        } else {
            const int i = threadIdx.x % LL, r0 = threadIdx.x / LL, dr = T / LL;
            if (i < q.nl) {
                const double *src = in + i + (long long)r0 * a.es;
#pragma unroll 4
                for (int r = r0; r < N; r += dr, src += dr * a.es) cp_async8(dst + r * LL + i + (r >> 4) * YP, src);
            }
        }
    };
    const bool blend_on = a.epi == EPI_BLEND;
    const int pc = min(p, P - 1);  // threads past the last block hold zero rows
    const bool two = a.nst == 2;
    int stage = 0;
    int t;
    // type of this thread's line, taken a tile ahead (its load is not waited for in the solve)
    auto type_of = [&](const Tile &q) { return a.ntypes > 1 && l < q.nl ? (int)a.ltype[q.L0 + l] : 0; };
    t = type_of(tile_of(job0));
    int staged = __shfl_sync(0xffffffffu, t, 0);  // lane 0 holds the first line
    stage_type(staged);
    int sb = c.blk[t * P + pc];
    // the coefficients do not depend on the launch before this one, the lines do
    pdl_wait();
    issue(tile_of(job0), lsm);
    const double blend = blend_on ? sweep_blend(a) : 0.0;
    for (int job = job0; job < a.njobs; job += jstep) {
    double *tl = lsm + stage * tsize;
    cp_async_wait_all();
    sync();  // the tile has landed, and the other stage's results have left
    const int ahead = job + jstep;
    int tnext = 0;
    if (ahead < a.njobs) {
        const Tile next = tile_of(ahead);
        tnext = type_of(next);
        if (two) issue(next, lsm + (stage ^ 1) * tsize);
    }
    const double *Qt = t == staged ? sc : c.Q + t * td;
    const double *Qr = Qt + pc * (M * Q6 + 2);

    auto at = [&](int r) { return XD ? l * pitch + r + (r >> 4) : r * LL + l + (r >> 4) * YP; };
    // row r of the line: cyclic lines wrap once, zero outside
    auto row = [&](int r) {
        if (PER) {
            r += r < 0 ? N : 0;
            r -= r >= N ? N : 0;
        }
        return r >= 0 && r < N ? tl[at(r)] : 0.0;
    };
    double w[M + 2 * H];
    double *const own = tl + at(sp);  // this block's rows: one pad between blocks
    constexpr int RS = XD ? 1 : LL, PS = XD ? 1 : YP;
    if (p < P) {
        if (sp + M <= N) {
#pragma unroll
            for (int j = 0; j < M; j++) w[H + j] = own[j * RS];
        } else {
#pragma unroll
            for (int j = 0; j < M; j++) w[H + j] = row(sp + j);
        }
        if (p > 0 && sp + M + H <= N) {
#pragma unroll
            for (int k = 0; k < H; k++) {
                w[k] = own[(k - H) * RS - PS];
                w[H + M + k] = own[(M + k) * RS + PS];
            }
        } else {
#pragma unroll
            for (int k = 0; k < H; k++) {
                w[k] = row(sp - H + k);
                w[H + M + k] = row(sp + M + k);
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < M + 2 * H; k++) w[k] = 0.0;
    }

    // ---- band product: the uniform band, or this block's own rows
    if (sb < 0) {
#pragma unroll
        for (int j = 0; j < M; j++) {
            double acc = c.band[NR - 1] * w[j + H];
#pragma unroll
            for (int q = 1; q < NR; q++) acc = acc + c.band[NR - 1 + q] * w[j + H + q] + c.band[NR - 1 - q] * w[j + H - q];
            w[j] = acc;
        }
        if (sp + M > N) {  // no rows past the line's end
#pragma unroll
            for (int j = 0; j < M; j++)
                if (sp + j >= N) w[j] = 0.0;
        }
    } else {
        const double *Rr = S + (size_t)sb * bd;
#pragma unroll
        for (int j = 0; j < M; j++) {
            double rc[W + 1];
            const double2 *r2 = reinterpret_cast<const double2 *>(Rr + j * WP);
#pragma unroll
            for (int v = 0; v < (W + 1) / 2; v++) {
                const double2 x = r2[v];
                rc[2 * v] = x.x;
                rc[2 * v + 1] = x.y;
            }
            double acc = rc[NR - 1] * w[j + H];
#pragma unroll
            for (int q = 1; q < NR; q++) acc = acc + rc[NR - 1 + q] * w[j + H + q] + rc[NR - 1 - q] * w[j + H - q];
            w[j] = acc;
        }
    }
    // ---- forward recurrence; cyclic: x(1) = D . rhs, corner terms, the reduced recurrence
    // (derivs.F90:786-799)
    double yprev = 0.0, x1 = 0.0;
    int jl = -1;
    double2 cc = make_double2(0.0, 0.0);
    if (PER) {
        double dot = 0.0;
#pragma unroll
        for (int j = 0; j < M; j++) dot = j == 0 ? w[0] * Qr[4] : dot + w[j] * Qr[j * Q6 + 4];
        if (p >= P) dot = 0.0;
        // a group's sum is (d0 + d2) + (d1 + d3)
        if constexpr (narrow) {
            dot = dot + __shfl_xor_sync(0xffffffffu, dot, 2 * LL);
            dot = dot + __shfl_xor_sync(0xffffffffu, dot, LL);
            if (sg == 0 && gi < ng) xs[gi * LL] = dot;
            sync();
            x1 = xs[0];
            for (int k = 1; k < ng; k++) x1 = x1 + xs[k * LL];
        } else {
            if (p < P) xs[p * LL] = dot;
            sync();
            if constexpr (!GROUPS) {
                x1 = xs[0];
                for (int k = 1; k < P; k++) x1 = x1 + xs[k * LL];
            }
            for (int k = 0; GROUPS && k < ng; k++) {
                double d[4];
#pragma unroll
                for (int q = 0; q < 4; q++) d[q] = 4 * k + q < P ? xs[(4 * k + q) * LL] : 0.0;
                const double g = (d[0] + d[2]) + (d[1] + d[3]);
                x1 = k ? x1 + g : g;
            }
        }
        cc = *reinterpret_cast<const double2 *>(Qt + td - 2);
        jl = N - 1 - sp;  // the line's last row in this block, if it is here
    }
#pragma unroll
    for (int j = 0; j < M; j++) {
        if (PER && j == 0 && p == 0) continue;  // row 0 is x(1)
        double g = w[j];
        if (PER && j == 1 && p == 0) g = g - cc.x * x1;
        if (PER && j == jl) g = g - cc.y * x1;
        const double2 ab = *reinterpret_cast<const double2 *>(Qr + j * Q6);
        const double y = (g - ab.x * yprev) * ab.y;
        w[j] = y;
        yprev = y;
    }
    if (PER && p == 0) w[0] = x1;

    // ---- value entering each block: y(start-1) = e + pe y(previous start-1), composed over the
    // blocks of a warp, then over the warps before it
    double Y = 0.0;
    {
        const double e = yprev, pe = Qr[(M - 1) * Q6 + 3];
        double yl = 0.0, pl = 1.0, Yw = 0.0;
        double *const se = xs + NS * LL, *const sp_ = xs + 2 * NS * LL;
        if constexpr (narrow) {
#pragma unroll
            for (int s = 1; s < 4; s++) {
                const double ue = __shfl_up_sync(0xffffffffu, e + pe * yl, LL), up = __shfl_up_sync(0xffffffffu, pe * pl, LL);
                if (sg == s) { yl = ue; pl = up; }
            }
            if (sg == 3 && gi < ng) {
                se[gi * LL] = e + pe * yl;
                sp_[gi * LL] = pe * pl;
            }
            sync();
            for (int k = 0; k < gi; k++) Yw = se[k * LL] + sp_[k * LL] * Yw;
        } else {
            if (p < P) {
                se[p * LL] = e;
                sp_[p * LL] = pe;
            }
            sync();
            if constexpr (!GROUPS)
                for (int k = 0; k < p; k++) Yw = se[k * LL] + sp_[k * LL] * Yw;
            for (int k = 0; GROUPS && k < gi; k++) {
                double ge = 0.0, gp = 1.0;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const double ek = se[(4 * k + q) * LL], pk = sp_[(4 * k + q) * LL];
                    ge = ek + pk * ge;
                    gp = pk * gp;
                }
                Yw = ge + gp * Yw;
            }
            for (int k = 4 * gi; GROUPS && k < p; k++) {
                const double ek = se[k * LL], pk = sp_[k * LL];
                yl = ek + pk * yl;
                pl = pk * pl;
            }
        }
        Y = yl + pl * Yw;
    }
    double xprev = 0.0;
#pragma unroll
    for (int j = M - 1; j >= 0; j--) {
        if (PER && j == 0 && p == 0) break;  // x(1) is final
        const double2 cp = *reinterpret_cast<const double2 *>(Qr + j * Q6 + 2);  // (bC, pi)
        const double y = w[j] + cp.y * Y;  // Y = 0 in the first block
        const double x = y - cp.x * xprev;
        w[j] = x;
        xprev = x;
    }
    double X = 0.0;
    {
        const double e = p < P ? xprev : 0.0, re = Qr[5];
        double xl = 0.0, pl = 1.0, Xw = 0.0;
        double *const se = xs + 3 * NS * LL, *const sr = xs + 4 * NS * LL;
        if constexpr (narrow) {
#pragma unroll
            for (int s = 2; s >= 0; s--) {
                const double ue = __shfl_down_sync(0xffffffffu, e + re * xl, LL), up = __shfl_down_sync(0xffffffffu, re * pl, LL);
                if (sg == s) { xl = ue; pl = up; }
            }
            if (sg == 0 && gi < ng) {
                se[gi * LL] = e + re * xl;
                sr[gi * LL] = re * pl;
            }
            sync();
            for (int k = ng - 1; k > gi; k--) Xw = se[k * LL] + sr[k * LL] * Xw;
        } else {
            if (p < P) {
                se[p * LL] = e;
                sr[p * LL] = re;
            }
            sync();
            if constexpr (!GROUPS)
                for (int k = P - 1; k > p; k--) Xw = se[k * LL] + sr[k * LL] * Xw;
            for (int k = ng - 1; GROUPS && k > gi; k--) {
                double ge = 0.0, gp = 1.0;
#pragma unroll
                for (int q = 3; q >= 0; q--) {
                    if (4 * k + q >= P) continue;
                    const double ek = se[(4 * k + q) * LL], rk = sr[(4 * k + q) * LL];
                    ge = ek + rk * ge;
                    gp = rk * gp;
                }
                Xw = ge + gp * Xw;
            }
            for (int k = min(4 * gi + 3, P - 1); GROUPS && k > p; k--) {
                const double ek = se[k * LL], rk = sr[k * LL];
                xl = ek + rk * xl;
                pl = rk * pl;
            }
        }
        X = xl + pl * Xw;
    }
#pragma unroll
    for (int j = 0; j < M; j++) {
        const double rho = Qr[j * Q6 + 5];
        w[j] = (PER && j == 0 && p == 0) ? w[0] : w[j] + rho * X;  // X = 0 in the last block
    }

    // ---- store, blended with the input that the tile still holds
    const Tile cur = tile_of(job);
    double *out = a.out + (long long)cur.b * a.out_bstride + (long long)a.out_slot[cur.f] * a.npts + cur.base;
    if (p < P && l < cur.nl) {
        if (blend_on) {
#pragma unroll
            for (int j = 0; j < M; j++) {
                const double o = sp + j < N ? own[j * RS] : 0.0;
                w[j] = o + blend * (w[j] - o);
            }
        }
        double *to = out + l + (long long)sp * a.es;
        if (sp + M <= N) {
#pragma unroll
            for (int j = 0; j < M; j++) {
                if (XD) own[j] = w[j];
                else { *to = w[j]; to += a.es; }
            }
        } else {
#pragma unroll
            for (int j = 0; j < M; j++) {
                if (sp + j >= N) continue;
                if (XD) own[j] = w[j];
                else to[(long long)j * a.es] = w[j];
            }
        }
    }
    if (XD) {
        sync();
        for (int n = warp; n < cur.nl; n += nw) {
            double *dst = out + (long long)n * N + lane;
            const double *src = tl + n * pitch + lane + (lane >> 4);
#pragma unroll 4
            for (int r = lane; r < N; r += 32, src += 34, dst += 32) *dst = *src;
        }
    }
    if (ahead < a.njobs) {
        if (two) stage ^= 1;
        else {
            sync();  // the stage has been read
            issue(tile_of(ahead), lsm);
        }
        t = tnext;
        sb = c.blk[t * P + pc];
        const int t0 = __shfl_sync(0xffffffffu, t, 0);
        if (t0 != staged) {  // the same decision in every warp
            sync();
            stage_type(t0);
            staged = t0;
        }
    }
    }
}

// One direction.
template <bool XD, bool PER, int NR, int LL>
__global__ void __launch_bounds__(line_bound(NR, LL))
    k_lsweep(const __grid_constant__ SweepArgs a, const __grid_constant__ LineArgs c)
{
    pdl_launch();
    line_run<XD, PER, NR, LL, false>(a, c, blockIdx.x, gridDim.x);
}

// The x sweep (the first nx CTAs) and the y sweep of a 2-D stage in one launch, LL-line tiles.
// Each is a fraction of a round on a small grid: one launch after another took 4.5 us each and
// two streams a fork and a join.  (Forming the stresses while the second sweeps load them, which
// would save a launch more, took 22 us a sweep against 11 and 2 for the stress kernel: each
// thread forms sixteen of them, a division and a square root apiece, before its solve.)
template <bool PERX, bool PERY, int NR, int LL>
__global__ void __launch_bounds__(line_bound(NR, LL))
    k_lsweep_xy(const __grid_constant__ SweepArgs ax, const __grid_constant__ LineArgs cx,
                const __grid_constant__ SweepArgs ay, const __grid_constant__ LineArgs cy, int nx)
{
    pdl_launch();
    if ((int)blockIdx.x < nx) line_run<true, PERX, NR, LL, true>(ax, cx, blockIdx.x, nx);
    else line_run<false, PERY, NR, LL, true>(ay, cy, blockIdx.x - nx, gridDim.x - nx);
}

// The instantiation for a direction, kind of line, band and lines per tile (4, 8, 16 or 32); null for
// bands outside 2..7.  Defined in lsweep_x.cu and lsweep_yz.cu.
void *line_kernel_x(bool per, int nR, int LL);
void *line_kernel_yz(bool per, int nR, int LL);
// k_lsweep_xy, tiles of 8 or 32 lines (lsweep_xy.cu)
void *line_kernel_xy(bool perx, bool pery, int nR, int LL);

template <bool XD, bool PER, int LL>
void *pick_line_kernel(int nR)
{
    switch (nR) {
    case 2: return (void *)k_lsweep<XD, PER, 2, LL>;
    case 3: return (void *)k_lsweep<XD, PER, 3, LL>;
    case 4: return (void *)k_lsweep<XD, PER, 4, LL>;
    case 5: return (void *)k_lsweep<XD, PER, 5, LL>;
    case 6: return (void *)k_lsweep<XD, PER, 6, LL>;
    case 7: return (void *)k_lsweep<XD, PER, 7, LL>;
    default: return nullptr;
    }
}

}  // namespace gatt
