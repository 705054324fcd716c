// ib_device.cuh -- device functions of the immersed boundary shared by the
// one-kernel-per-stage launches (ib_kernels.cu) and the step loop
// (step_loop.cu). Both call the same functions in the same order, so a step's
// results do not depend on which of them ran it.
#pragma once
#include "lbm_internal.h"
#include "lbm_node.cuh"

namespace lbm_ib {

constexpr int BS = 16;                 // block size of the cyclic reduction
constexpr int NMARK_MAX = 2048;        // largest marker count
constexpr int FL = 2 * BS;             // columns of a coupling panel [L_o | L_q^T]
constexpr int GW = 3 * BS;             // row width of a stored factor block [D^-1 | F_L | F_U]
constexpr int GP = BS + 1;             // padded row stride of square blocks in shared memory
constexpr int NPART = 3 * LBM_MAXW + 3;   // per-tile partials of the force sums
constexpr int TILE = 16;                  // correction-patch tile (nodes per side)
constexpr int TILE_CAP = 256;             // markers listed per tile
constexpr int TILE_THREADS = TILE * TILE;

// A right-hand side or solution value that has not been computed: a NaN whose
// payload no arithmetic produces (results are canonical NaNs or carry an
// operand's payload, and no operand has this one; is_value() turns it into
// the canonical NaN should a result ever hold it).
#define LBM_NOT_YET 0xfff8d2a9c0debeefull
__device__ __forceinline__ double not_yet() { return __longlong_as_double((long long)LBM_NOT_YET); }
__device__ __forceinline__ double is_value(double x)
{
    return __double_as_longlong(x) == (long long)LBM_NOT_YET ? __longlong_as_double(0x7ff8000000000000ll) : x;
}

// FP64 moments of the streamed populations at an interior node
template <typename T, typename LD = LdNc>
__device__ __forceinline__ void node_moments(const IBArgs &a, const T *fin, int i, int j, double &rho, double &u, double &v)
{
    double g[9];
#pragma unroll
    for (int k = 0; k < 9; ++k)
        g[k] = (double)Store<T>::cvt(LD::ld(fin + (long long)k * a.plane + (long long)(j - lbm_ey(k)) * a.pitch +
                                            (i - lbm_ex(k))));
    const double drho = ((g[0] + g[1]) + (g[2] + g[3])) + ((g[4] + g[5]) + (g[6] + g[7])) + g[8];
    const double jx = (g[1] - g[3]) + (g[5] - g[6]) + (g[8] - g[7]);
    const double jy = (g[2] - g[4]) + (g[5] + g[6]) - (g[7] + g[8]);
    rho = 1.0 + drho;
    u = jx / rho;
    v = jy / rho;
}

__device__ __forceinline__ const double *motion_row(const IBArgs &a, int step_index, double *time_out)
{
    const double time = (double)(step_index - 1) * (a.scale * a.uu);   // solution.f90:289
    int idx = (int)llround(time / a.mdt) + 1;                             // mode.f90:280-281
    idx = idx < 1 ? 1 : (idx > a.msteps ? a.msteps : idx);
    if (time_out) *time_out = time;
    return a.mstep + (long long)(idx - 1) * a.mcols;
}

__device__ __forceinline__ int4 mbox(const Marker &m) { return make_int4(m.i1, m.i2, m.j1, m.j2); }

// a marker as make_marker leaves it: support box within bounds (an empty
// box included) and a wing index of the case
__device__ __forceinline__ bool marker_ok(const IBArgs &a, const Marker &m)
{
    return box_in_bounds(m.i1, m.i2, m.j1, m.j2, a.nx, a.ny) && m.wing >= 0 && m.wing < a.nwing;
}

// marker at position s of the solve order, or -1 (and the kernel's status
// bit set) when the order holds an index outside the markers
__device__ __forceinline__ int order_at(const IBArgs &a, int s, unsigned bit)
{
    const int k = a.perm[s];
    if (k < 0 || k >= a.nseg) {
        atomicOr(a.status, bit);
        return -1;
    }
    return k;
}

// tiles of the patch grid (the tile lists of one slot)
__device__ __forceinline__ int patch_tiles(const IBArgs &a) { return (int)(a.st_tiles / (TILE_CAP + 1)); }

// time and motion columns of this step's force.dat row (solution.f90:350-375)
__device__ __forceinline__ void write_header(const IBArgs &a, const double *row, double time, int ring_slot)
{
    double *fr = a.force_ring + (long long)ring_slot * a.row_len;
    fr[0] = time;
    const int mc = 1 + 3 * a.nwing + 3;
    for (int w = 0; w < a.nwing; ++w) {
        const double *r = row + 1 + 9 * w;   // angle omega omgac sa sau saac sb sbv sbac
        double *o = fr + mc + 9 * w;         // solution.f90:363-374 order
        o[0] = r[3]; o[1] = r[4]; o[2] = r[5]; o[3] = r[6]; o[4] = r[7]; o[5] = r[8];
        o[6] = r[0]; o[7] = r[1]; o[8] = r[2];
    }
}

// Arguments of a later step of the same handle from those of slot 0
// (make_args): the step's buffer slot holds its geometry, its factorization
// and its own right-hand sides, solution, tile partials and residual.
__device__ __forceinline__ IBArgs step_args(IBArgs a, int step)
{
    const int slot = step % a.nslots;
    a.mk += slot * a.st_mk;
    a.perm += slot * a.st_perm;
    a.key += slot * a.st_perm;
    a.B += slot * a.st_B;
    a.gf += slot * a.wk_gf;
    a.pinfo += slot;
    a.tiles += slot * a.st_tiles;
    a.ctile += slot * (a.st_tiles / (TILE_CAP + 1));
    a.nsup += slot;
    a.fmode += 2 * slot;
    a.fstatus += slot;
    a.rhs += slot * a.st_rhs;
    a.y += slot * a.st_rhs;
    a.partial += slot * a.st_part;
    a.solve_res += 2 * slot;
    a.cur_step = step;
    return a;
}

// One warp's interpolation of a marker, b = D u* over its support box: the
// nodes and weights of the lane, from the marker's geometry ...
struct InterpLane {
    int i0, j0, i1, j1;   // at most LBM_BOX^2 = 36 nodes: lane t takes nodes t and t + 32
    bool h0, h1;          // the lane has a first, a second node
    double w0, w1;        // X1(k,i) = kernel1*kernel2 (:1602)
    double ub, vb;
    int pos;              // where its right-hand sides go (-1: nowhere)
};

__device__ __forceinline__ InterpLane interp_lane(const IBArgs &a, int k, int lane)
{
    // the marker's box and kernel values are read where they lie (a local
    // copy of the struct, indexed by node, would live on the stack)
    const Marker *mp = a.mk + k;
    const int i1 = mp->i1, i2 = mp->i2, j1 = mp->j1, j2 = mp->j2;
    const bool ok = box_in_bounds(i1, i2, j1, j2, a.nx, a.ny);
    if (!ok && lane == 0) atomicOr(a.status, LBM_ST_INDEX_INTERP);
    const int nbx = ok ? i2 - i1 + 1 : 0, nby = ok ? j2 - j1 + 1 : 0;
    const int nn = nbx > 0 && nby > 0 ? nbx * nby : 0;
    InterpLane l;
    l.ub = mp->ub;
    l.vb = mp->vb;
    l.pos = mp->pos;
    if (l.pos < 0 || l.pos >= a.nseg) {
        if (lane == 0) atomicOr(a.status, LBM_ST_INDEX_INTERP);
        l.pos = -1;
    }
    // rows of a node number: n / nbx for n < 64 and nbx <= 6, exact
    const float rn = nn > 0 ? __frcp_rn((float)nbx) : 0.0f;
    const int r0 = (int)(((float)lane + 0.5f) * rn), r1 = (int)(((float)lane + 32.5f) * rn);
    const int c0 = lane - r0 * nbx, c1 = lane + 32 - r1 * nbx;
    // a lane without a node of its own loads the box's first and leaves it
    // out; with an empty box every lane loads an interior node of the lattice
    const bool h0 = lane < nn, h1 = lane + 32 < nn;
    l.h0 = h0;
    l.h1 = h1;
    const int bi = nn > 0 ? i1 : 1, bj = nn > 0 ? j1 : 1;
    l.i0 = h0 ? bi + c0 : bi;
    l.j0 = h0 ? bj + r0 : bj;
    l.i1 = h1 ? bi + c1 : l.i0;
    l.j1 = h1 ? bj + r1 : l.j0;
    l.w0 = h0 ? rmul(mp->phx[c0], mp->phy[r0]) : 0.0;
    l.w1 = h1 ? rmul(mp->phx[c1], mp->phy[r1]) : 0.0;
    return l;
}

// ... and the sum over both nodes' velocities (all loads issued before the
// first use) and over the lanes: U_b - b in lane 0 (comj, :1624-1629)
template <typename T, typename LD>
__device__ __forceinline__ void interp_sum(const IBArgs &a, const T *fin, const InterpLane &l, double &ru, double &rv)
{
    double rho0, u0, v0, rho1, u1, v1;
    node_moments<T, LD>(a, fin, l.i0, l.j0, rho0, u0, v0);
    node_moments<T, LD>(a, fin, l.i1, l.j1, rho1, u1, v1);
    double su = l.h0 ? rfma(l.w0, u0, 0.0) : 0.0, sv = l.h0 ? rfma(l.w0, v0, 0.0) : 0.0;
    if (l.h1) {
        su = rfma(l.w1, u1, su);
        sv = rfma(l.w1, v1, sv);
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        su += __shfl_down_sync(0xffffffffu, su, off);
        sv += __shfl_down_sync(0xffffffffu, sv, off);
    }
    ru = l.ub - su;
    rv = l.vb - sv;
}

// dense fallback, solve: L z = r, then L^T y = z, for the two right-hand
// sides yv[0..n) and yv[n..2n) (shared memory), the nt threads of a CTA
static __device__ void dense_tri(const IBArgs &a, double *yv, int nt)
{
    const int n = a.nseg, tid = threadIdx.x;
    const double *L = a.B;
    for (int k = 0; k < n; ++k) {
        const double dk = L[(long long)k * n + k];
        const double z0 = yv[k] / dk, z1 = yv[n + k] / dk;
        __syncthreads();
        if (tid == 0) { yv[k] = z0; yv[n + k] = z1; }
        for (int i = k + 1 + tid; i < n; i += nt) {
            const double lik = L[(long long)i * n + k];
            yv[i] -= lik * z0;
            yv[n + i] -= lik * z1;
        }
        __syncthreads();
    }
    for (int j = n - 1; j >= 0; --j) {
        if (tid < 2) yv[tid * n + j] /= L[(long long)j * n + j];
        __syncthreads();
        for (int q = tid; q < 2 * j; q += nt) {
            const int c = q / j, i = q % j;
            yv[c * n + i] -= L[(long long)j * n + i] * yv[c * n + j];
        }
        __syncthreads();
    }
}

// ---- one warp's share of a level of the cyclic-reduction sweeps ------------
// Lane i + 16 c owns row i of the block for right-hand side c; X holds the
// pairs (right-hand side 0, 1) in the solve order. Each sum is one chain in
// column order: with 2-byte storage the flow amplifies a change in the last
// bits of the solution to the storage's own rounding level, so the order is
// part of what a run gives.

// even block e: r_e -= F_L(q)^T r_q + F_U(p)^T r_p, q = e + st, p = e - st
__device__ __forceinline__ void bcr_forward(const double *Fq, const double *Fp, double *X, int e, int st, bool has_q,
                                            bool has_p, int lane)
{
    const int i = lane & (BS - 1), c = lane >> 4;
    double acc = 0.0;
    if (has_q) {
        const double *F = Fq + BS + i;       // F_L(q)[t][i]
        const double *r = X + 2 * (e + st) * BS + c;
#pragma unroll
        for (int t = 0; t < BS; ++t) acc = rfma(F[t * GW], r[2 * t], acc);
    }
    if (has_p) {
        const double *F = Fp + 2 * BS + i;   // F_U(p)[t][i]
        const double *r = X + 2 * (e - st) * BS + c;
#pragma unroll
        for (int t = 0; t < BS; ++t) acc = rfma(F[t * GW], r[2 * t], acc);
    }
    X[2 * (e * BS + i) + c] -= acc;
}

// odd block o: x_o = D_o^-1 r_o - F_L(o) x_p - F_U(o) x_q. The rows of a
// block lie GW = 96 words apart, all on one bank: lane row i starts at column
// i, so that the 16 rows read in one step fall on distinct banks.
__device__ __forceinline__ void bcr_backward(const double *Gb, double *X, int o, int st, bool has_q, int lane)
{
    const int i = lane & (BS - 1), c = lane >> 4;
    const double *G = Gb + i * GW;
    const double *ro = X + 2 * o * BS + c, *rp = X + 2 * (o - st) * BS + c, *rq = X + 2 * (o + st) * BS + c;
    double s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
    for (int t0 = 0; t0 < BS; ++t0) {
        const int t = (t0 + i) & (BS - 1);
        s1 = rfma(G[t], ro[2 * t], s1);
        s2 = rfma(G[BS + t], rp[2 * t], s2);
        if (has_q) s3 = rfma(G[2 * BS + t], rq[2 * t], s3);
    }
    __syncwarp();   // the block's right-hand sides are read before they are overwritten
    X[2 * (o * BS + i) + c] = s1 - s2 - s3;
}

// block 0, the last one left: x_0 = D_0^-1 r_0, rows of D_0^-1 ld apart
__device__ __forceinline__ void bcr_root(const double *D, int ld, double *X, int lane)
{
    const int i = lane & (BS - 1), c = lane >> 4;
    const double *G = D + i * ld;
    double x = 0.0;
#pragma unroll
    for (int t = 0; t < BS; ++t) x = rfma(G[t], X[2 * t + c], x);
    __syncwarp();
    X[2 * i + c] = x;
}

// The solution of the marker at position pos after ib_solve, which leaves the
// odd blocks of the first level, half of all, to whoever needs them: their back
// substitution (bcr_backward's) waits for nothing but the even blocks, and the
// tiles have the threads for it. Eight lanes a marker (8 m .. 8 m + 7 of the
// warp): lane 2 p + c takes sum p of component c; the lanes 0 and 1 return the
// components, and store them for the residual check.
__device__ __forceinline__ double marker_solution(const IBArgs &a, int pos, int lane)
{
    const int c = lane & 1, part = (lane >> 1) & 3;
    const int o = pos / BS, i = pos % BS, nb = (a.nseg + BS - 1) / BS;
    const bool odd = pos >= 0 && (o & 1) && !a.fmode[0];
    double s = 0.0;
    if (odd && part < 3) {
        const int blk = part == 0 ? o : part == 1 ? o - 1 : o + 1;
        const double *G = a.gf + ((long long)o * BS + i) * GW + part * BS;
        const double *x = (part == 0 ? a.rhs : a.y) + 2 * blk * BS + c;
        const int m = blk < nb ? a.nseg - blk * BS : 0;   // past the end: 0
        if (m >= BS) {
#pragma unroll
            for (int t0 = 0; t0 < BS; ++t0) {
                const int t = (t0 + i) & (BS - 1);
                s = rfma(G[t], x[2 * t], s);
            }
        } else if (blk < nb) {
#pragma unroll
            for (int t0 = 0; t0 < BS; ++t0) {
                const int t = (t0 + i) & (BS - 1);
                s = rfma(G[t], t < m ? x[2 * t] : 0.0, s);
            }
        }
    }
    const double s2 = __shfl_down_sync(0xffffffffu, s, 2, 8), s3 = __shfl_down_sync(0xffffffffu, s, 4, 8);
    if (part != 0 || pos < 0) return 0.0;
    if (!odd) return a.y[2 * pos + c];
    const double x = s - s2 - s3;
    a.y[2 * pos + c] = x;
    return x;
}

// ---- a correction tile (TILE_THREADS threads) --------------------------------

struct TileSmem {
    // markers whose support box meets the tile, in marker order
    int4 box[TILE_THREADS];
    double ph[TILE_THREADS][12];
    double y[TILE_THREADS][2];
    int wing[TILE_THREADS];
    double red[8][NPART];
    int wsum[8];
    int nlist;
};

// marker k into place t of the staged list, without its solution values; an
// index outside the markers is reported and leaves an empty box
__device__ __forceinline__ bool tile_stage(const IBArgs &a, TileSmem &S, int t, int k)
{
    if (k >= 0 && k < a.nseg && marker_ok(a, a.mk[k])) {
        const Marker &m = a.mk[k];
        S.box[t] = mbox(m);
#pragma unroll
        for (int q = 0; q < 6; ++q) { S.ph[t][q] = m.phx[q]; S.ph[t][6 + q] = m.phy[q]; }
        S.wing[t] = m.wing;
        return true;
    }
    atomicOr(a.status, LBM_ST_INDEX_TILE);
    S.box[t] = make_int4(1, 0, 1, 0);
    S.wing[t] = 0;
    return false;
}

// the position of listed marker k in the solve order (-1 and a report where
// the list or the marker holds an index out of range)
__device__ __forceinline__ int tile_position(const IBArgs &a, int k)
{
    const int pos = k >= 0 && k < a.nseg ? a.mk[k].pos : -1;
    if (pos >= 0 && pos < a.nseg) return pos;
    atomicOr(a.status, LBM_ST_INDEX_TILE);
    return -1;
}

// the solution of the n markers of a staged list (marker(t): its t-th), by
// the tile's threads
template <class F>
__device__ __forceinline__ void tile_solve(const IBArgs &a, TileSmem &S, int n, int th, F marker)
{
    const int lane = th & 31;
    for (int m0 = 0; m0 < n; m0 += TILE_THREADS / 8) {
        const int t = m0 + (th >> 3);
        const double x = marker_solution(a, t < n ? tile_position(a, marker(t)) : -1, lane);
        if (t < n && (lane & 7) < 2) S.y[t][lane & 1] = x;
    }
}

// du = D^T y at node (gi, gj) from the staged markers first .. n-1, in marker order;
// wing: the lowest wing whose support box holds the node
__device__ __forceinline__ void tile_gather(const TileSmem &S, int first, int n, int gi, int gj, double &du, double &dv,
                                            int &wing)
{
    for (int t = first; t < n; ++t) {
        const int4 b = S.box[t];
        if (gi >= b.x && gi <= b.y && gj >= b.z && gj <= b.w) {
            const double wgt = rmul(S.ph[t][gi - b.x], S.ph[t][6 + gj - b.z]);
            du = rfma(wgt, S.y[t][0], du);
            dv = rfma(wgt, S.y[t][1], dv);
            wing = min(wing, S.wing[t]);
        }
    }
}

// The same in two parts, for when the solution comes later than the rest: the
// covering markers of the thread's node (their number is returned) with the
// first TILE_KEEP weights, and the sum over them.
constexpr int TILE_KEEP = 16;
struct TileWeights {
    double w[TILE_KEEP][TILE_THREADS];
    unsigned char at[TILE_KEEP][TILE_THREADS];
};
__device__ __forceinline__ int tile_cover(const TileSmem &S, TileWeights &W, int n, bool active, int gi, int gj, int th,
                                          int &wing)
{
    // a warp's nodes are two rows of the tile: its lanes first find the
    // markers that meet them
    const int lane = th & 31, j0 = gj - (lane >> 4);
    int cnt = 0;
    for (int t0 = 0; t0 < n; t0 += 32) {
        int4 b = make_int4(1, 0, 1, 0);
        if (t0 + lane < n) b = S.box[t0 + lane];
        unsigned m = __ballot_sync(0xffffffffu, b.z <= j0 + 1 && b.w >= j0);
        while (m) {
            const int t = t0 + __ffs((int)m) - 1;
            m &= m - 1;
            const int4 q = S.box[t];
            if (active && gi >= q.x && gi <= q.y && gj >= q.z && gj <= q.w) {
                if (cnt < TILE_KEEP) {
                    W.w[cnt][th] = rmul(S.ph[t][gi - q.x], S.ph[t][6 + gj - q.z]);
                    W.at[cnt][th] = (unsigned char)t;
                }
                ++cnt;
                wing = min(wing, S.wing[t]);
            }
        }
    }
    return cnt;
}
__device__ __forceinline__ void tile_sum(const TileSmem &S, const TileWeights &W, int cnt, int n, int gi, int gj, int th,
                                         double &du, double &dv)
{
    const int m = min(cnt, TILE_KEEP);
#pragma unroll 4
    for (int c = 0; c < m; ++c) {
        const double w = W.w[c][th];
        const int t = W.at[c][th];
        du = rfma(w, S.y[t][0], du);
        dv = rfma(w, S.y[t][1], dv);
    }
    int wing = 0;
    if (cnt > TILE_KEEP) tile_gather(S, W.at[TILE_KEEP - 1][th] + 1, n, gi, gj, du, dv, wing);
}

// force and moment of a support node of `wing` (boundary_condition.f90:
// 1661-1675) from its streamed populations and its velocity correction
template <typename C>
__device__ __forceinline__ void node_force(const IBArgs &a, const double *row, const C g[9], int gi, int gj, int wing,
                                           double du, double dv, double &fx, double &fy, double &mz)
{
    // FP64 density of the streamed populations
    const double drho = (((double)g[0] + (double)g[1]) + ((double)g[2] + (double)g[3])) +
                        (((double)g[4] + (double)g[5]) + ((double)g[6] + (double)g[7])) + (double)g[8];
    const double rho = 1.0 + drho;
    const double temp1 = rmul(rmul(2.0, rho), du), temp2 = rmul(rmul(2.0, rho), dv);
    const double sa = row[4 + 9 * wing], sb = row[7 + 9 * wing];
    fx = -temp1;
    fy = -temp2;
    const double x0 = (rfma(a.scale, (double)gi, a.ox) - (a.xc + sa)) / a.scale;
    const double y0 = (rfma(a.scale, (double)gj, a.oy) - (a.yc + sb)) / a.scale;
    mz = rfma(y0, temp1, rmul(-x0, temp2));
}

// the warps' sums of the nodes' forces per wing into S.red (warp: 0..7 of the
// tile); after a barrier of the tile's threads, tile_force_store adds them in
// warp order into the tile's partials
__device__ __forceinline__ void tile_force_warp(const IBArgs &a, TileSmem &S, bool in_support, int wing, double fx,
                                                double fy, double mz, int warp, int lane)
{
    for (int w = 0; w < a.nwing; ++w) {
        double v0 = (in_support && wing == w) ? fx : 0.0;
        double v1 = (in_support && wing == w) ? fy : 0.0;
        double v2 = (in_support && wing == w) ? mz : 0.0;
#pragma unroll
        for (int off = 16; off; off >>= 1) {
            v0 += __shfl_down_sync(0xffffffffu, v0, off);
            v1 += __shfl_down_sync(0xffffffffu, v1, off);
            v2 += __shfl_down_sync(0xffffffffu, v2, off);
        }
        if (lane == 0) { S.red[warp][3 * w] = v0; S.red[warp][3 * w + 1] = v1; S.red[warp][3 * w + 2] = v2; }
    }
}

__device__ __forceinline__ void tile_force_store(const IBArgs &a, const TileSmem &S, int tile, int t)
{
    if (t < 3 * a.nwing) {
        double sum = 0.0;
        for (int w8 = 0; w8 < 8; ++w8) sum += S.red[w8][t];
        a.partial[(long long)tile * NPART + t] = sum;
    }
}

}  // namespace lbm_ib
