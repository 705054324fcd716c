// ib_kernels.cu -- immersed boundary of one time step (FP64), ahead of the
// lattice update of the correction patch.
//
// Reference: move_boundary (airfoil.f90:244-338) and immersed_boundary_Wu
// (boundary_condition.f90:1512-1736). The reference builds dense X1 (nseg x
// nadj) and X2 = X1^T W (W = diag(arc_l)), forms A = X1 X2 with cublasDgemm,
// solves A x = U_b - X1 u* by LU (cusolverDnDgetrf/getrs) and spreads
// du = X2 x. With D = X1, A = (D D^T) W, so y = W x solves the symmetric
// positive definite system (D D^T) y = U_b - D u* and du = D^T y: the same
// correction, with arc_l dropping out.
//
// The marker positions follow the prescribed motion, so D D^T and its
// factorization depend on the step index only, not on the flow. The
// launches are therefore two chains. The factorization chain of a step
// (which the host runs a batch of steps ahead, beside the steps of the batch
// before, into the slots of the other half):
//   ib_geometry one thread per marker: position, boundary velocity, support
//               box and one-axis kernel values (move_boundary, :1540-1606);
//   ib_order    (several bodies only) one CTA sorts the markers along the
//               longer axis of the marker cloud. A single rigid body keeps one
//               order for the whole run: its markers sorted by body-frame
//               chordwise position, computed once on the host;
//   ib_assemble one CTA per 16-marker block of that order: D D^T is banded in
//               it (delta supports overlap only for markers less than 5 lu
//               apart per axis), so the CTA builds its diagonal block and the
//               block coupling it to the previous one, and checks that no
//               coupling reaches further;
//   ib_tile_scatter, ib_tile_sort  per 16 x 16 tile of the patch
//               rectangle, the markers whose support box meets it (each
//               marker appends itself; each tile sorts its list);
//   ib_factor   one CTA: correction-patch rectangle, then block cyclic
//               reduction of the block tridiagonal matrix (log2 of the block
//               count levels of Gauss-Jordan block inverses and block
//               products, FP64), keeping per eliminated block D^-1 and the two
//               coupling factors; a dense Cholesky replaces it when a coupling
//               reaches past the neighbouring block.
// The flow chain of the step:
//   ib_interp   one warp per marker: b = D u* over the support box and
//               rhs = U_b - b (:1609-1629);
//   ib_solve    one CTA: the forward and backward sweeps of the reduction
//               over the two right-hand sides, the factor blocks of the
//               levels above the first in shared memory, down to the odd
//               blocks of the first level, which the tiles that need them
//               solve (or the two triangular solves of the dense factor);
//   ib_tile_update  one CTA per correction tile (a 16 x 16 tile of the
//               patch rectangle that lists a marker): du = D^T y per node,
//               gathered in marker order (no atomics), the lattice update of
//               the tile's nodes with that correction, and the force and
//               moment sums (:1645-1675, solution.f90:327-336) in FP64 with a
//               deterministic two-level reduction. The lattice kernel skips
//               these nodes and updates all others;
//   ib_checks   the force row from the tiles' partials and the solve's
//               residual, after the step's update (ib_forces and ib_residual
//               in batches that run stage by stage).

#include <math.h>

#include "ib_device.cuh"

namespace {

using namespace lbm_ib;

#ifndef LBM_FACTOR_THREADS
#define LBM_FACTOR_THREADS 512
#endif
#ifndef LBM_SOLVE_THREADS
#define LBM_SOLVE_THREADS 512
#endif
#ifndef LBM_SOLVE_SMEM
#define LBM_SOLVE_SMEM 232192
#endif
constexpr int FACTOR_THREADS = LBM_FACTOR_THREADS;
constexpr int BOPS_WARPS = FACTOR_THREADS / 32;   // warps running block operations
constexpr int SOLVE_THREADS = LBM_SOLVE_THREADS;
constexpr int SOLVE_SMEM_BUDGET = LBM_SOLVE_SMEM;   // dynamic shared memory of ib_solve (bytes)

// Levels of the reduction whose factor blocks ib_solve keeps in shared memory:
// those from st0 on (the blocks that are multiples of st0, at index o / st0).
// Level 1's are read once, in the forward sweep, and stay in L2, so that a
// solve of 512 markers takes half an SM's shared memory.
// shared memory of a solve of nb blocks that keeps the levels from st on
__host__ __device__ constexpr int solve_bytes(int nb, int st)
{
    return ((nb + st - 1) / st * BS * GW + 2 * nb * BS) * (int)sizeof(double) + 16;
}
__host__ __device__ constexpr int solve_st0(int nb)
{
    int st = 2;
    while (solve_bytes(nb, st) > SOLVE_SMEM_BUDGET) st *= 2;
    return st;
}
constexpr int WS = BS * GP + BS * FL + BS * GP;   // workspace per warp (doubles)

// one-axis kernel value (boundary_condition.f90:1563-1600), disr = |r|
__device__ __forceinline__ double delta1(double disr, int smooth)
{
    const double pai = 3.1415926535897932384626433832795;
    if (smooth == 0) {
        if (fabs(disr) < 1.0)
            return 0.125 * (3.0 - 2.0 * fabs(disr) + sqrt(1.0 + 4.0 * fabs(disr) - 4.0 * disr * disr));
        else if ((fabs(disr) < 2.0) && (fabs(disr) >= 1.0))
            return 0.125 * (5.0 - 2.0 * fabs(disr) - sqrt(-7.0 + 12.0 * fabs(disr) - 4.0 * disr * disr));
        return 0.0;
    }
    if (fabs(disr) <= 0.5)
        return 0.375 + 0.03125 * pai - 0.25 * disr * disr;
    else if ((fabs(disr) <= 1.5) && (fabs(disr) >= 0.5))
        return 0.25 + 0.125 * (1.0 - disr) * sqrt(-2.0 + 8.0 * disr - 4.0 * disr * disr) -
               0.125 * asin(sqrt(2.0) * (disr - 1.0));
    else if ((fabs(disr) <= 2.5) && (fabs(disr) >= 1.5))
        return 1.0625 - 0.015625 * pai - 0.75 * disr + 0.125 * disr * disr +
               0.0625 * (disr - 2.0) * sqrt(-14.0 + 16.0 * disr - 4.0 * disr * disr) +
               0.0625 * asin(sqrt(2.0) * (disr - 2.0));
    return 0.0;
}


// Step of this CTA's member of a factorization launch: step0 + blockIdx.y,
// or per case in batched launches (the case's own start and count; -1 for
// the members past its count).
template <bool BATCH> __device__ __forceinline__ int factor_step(const IBArgs &base, int step0)
{
    if (!BATCH) return step0 + (int)blockIdx.y;
    return (int)blockIdx.y < base.fcount ? base.fstep0 + (int)blockIdx.y : -1;
}

// Arguments of one member of a batched factorization launch: the step
// step0 + blockIdx.y, its buffer slot (step modulo the slot count) and the
// member's working set.
__device__ __forceinline__ IBArgs member_args(IBArgs a, int step)
{
    const int slot = step % a.nslots, mem = blockIdx.y;
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
    a.status = a.fstatus;   // errors of the chain are reported by the step that uses it
    a.bD += mem * a.wk_blocks;
    a.bL += mem * a.wk_blocks;
    a.wmax += mem;
    return a;
}

// marker geometry of segment k (airfoil.f90:255-335, boundary_condition.f90:1540-1606)
__device__ Marker make_marker(const IBArgs &a, const double *row, int k)
{
    const double scale = a.scale, ox = a.ox, oy = a.oy;
    const int w = k / a.spw;
    const int p0 = w * a.ppw + (k - w * a.spw);
    const double angle = row[1 + 9 * w], omega = row[2 + 9 * w];
    const double sa = row[4 + 9 * w], sau = row[5 + 9 * w];
    const double sb = row[7 + 9 * w], sbv = row[8 + 9 * w];
    const double ca = cos(angle), sn = sin(angle);
    // airfoil.f90:261-263 (body_extra_s and movenum are zero: no dynamics)
    const double xa = ca * a.xb0[p0] + sn * a.yb0[p0] + sa + a.xc;
    const double xb = ca * a.xb0[p0 + 1] + sn * a.yb0[p0 + 1] + sa + a.xc;
    const double ya = -sn * a.xb0[p0] + ca * a.yb0[p0] + sb + a.yc;
    const double yb = -sn * a.xb0[p0 + 1] + ca * a.yb0[p0 + 1] + sb + a.yc;
    Marker m;
    m.xm = 0.5 * (xb + xa);                                           // :267-270
    m.ym = 0.5 * (yb + ya);
    // boundary_condition.f90:1547-1550 (body_extra_v is zero)
    m.ub = a.uu * (-omega * sn * 0.5 * (a.xb0[p0 + 1] + a.xb0[p0]) +
                   omega * ca * 0.5 * (a.yb0[p0 + 1] + a.yb0[p0]) + sau);
    m.vb = a.uu * (-omega * ca * 0.5 * (a.xb0[p0 + 1] + a.xb0[p0]) -
                   omega * sn * 0.5 * (a.yb0[p0 + 1] + a.yb0[p0]) + sbv);
    m.wing = w;
    m.pos = -1;
    for (int t = 0; t < LBM_BOX; ++t) m.phx[t] = m.phy[t] = 0.0;
    m.i1 = 3; m.i2 = 2; m.j1 = 3; m.j2 = 2;   // empty box unless set below
    // a marker off the lattice (or not finite) is a range error before any scan
    const double fx = (m.xm - ox) / scale + 1.0, fy = (m.ym - oy) / scale + 1.0;
    if (!(fx > 3.0 && fx < (double)(a.nx - 2) && fy > 3.0 && fy < (double)(a.ny - 2))) {
        atomicOr(a.status, LBM_ST_RANGE);
        return m;
    }
    // support box, 1-based scans of airfoil.f90:290-321
    int i1 = (int)((m.xm - ox) / scale + 1.0);
    for (int i = i1; i >= 1; --i)
        if (fabs((ox + (double)(i - 1) * scale - m.xm) / scale) > 2.5) { i1 = i + 1; break; }
    int i2 = (int)((m.xm - ox) / scale + 1.0);
    for (int i = i2; i <= a.nx; ++i)
        if (fabs((ox + (double)(i - 1) * scale - m.xm) / scale) > 2.5) { i2 = i - 1; break; }
    int j2 = (int)((m.ym - oy) / scale + 1.0);
    for (int i = j2; i <= a.ny; ++i)
        if (fabs((oy + (double)(i - 1) * scale - m.ym) / scale) > 2.5) { j2 = i - 1; break; }
    int j1 = (int)((m.ym - oy) / scale + 1.0);
    for (int i = j1; i >= 1; --i)
        if (fabs((oy + (double)(i - 1) * scale - m.ym) / scale) > 2.5) { j1 = i + 1; break; }
    if (i1 < 4 || j1 < 4 || i2 > a.nx - 3 || j2 > a.ny - 3 || i2 - i1 >= LBM_BOX || j2 - j1 >= LBM_BOX) {
        atomicOr(a.status, LBM_ST_RANGE);
        return m;
    }
    for (int t = 0; t < LBM_BOX; ++t) {
        const int ii = i1 + t, jj = j1 + t;
        m.phx[t] = ii <= i2 ? delta1(fabs((ox + scale * (double)(ii - 1) - m.xm) / scale), a.smooth) : 0.0;
        m.phy[t] = jj <= j2 ? delta1(fabs((oy + scale * (double)(jj - 1) - m.ym) / scale), a.smooth) : 0.0;
    }
    m.i1 = i1 - 1; m.i2 = i2 - 1; m.j1 = j1 - 1; m.j2 = j2 - 1;
    return m;
}


// one thread per marker: geometry of this step (errors go to the slot's status)
template <bool BATCH>
__global__ void __launch_bounds__(128) ib_geometry(const IBArgs base0, const IBArgs *batch, int step0)
{
    const IBArgs &base = BATCH ? batch[blockIdx.z] : base0;
    const int step_index = factor_step<BATCH>(base, step0);
    if (step_index < 0) return;
    const IBArgs a = member_args(base, step_index);
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.nseg) return;
    const double *row = motion_row(a, step_index, nullptr);
    a.mk[k] = make_marker(a, row, k);
    // the step's right-hand sides and solution are not there yet (the step
    // loop's CTAs wait for the values themselves)
    a.rhs[2 * k] = a.rhs[2 * k + 1] = not_yet();
    a.y[2 * k] = a.y[2 * k + 1] = not_yet();
}

// one warp per marker: b = D u* over the support box, rhs = U_b - b
template <typename T, bool BATCH>
__global__ void __launch_bounds__(256) ib_interp(const IBArgs a0, const IBArgs *batch)
{
    const IBArgs &a = BATCH ? batch[blockIdx.z] : a0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // bring the slot's factor blocks, which the lattice kernels have evicted
    // since the factorization wrote them, back into L2 for ib_solve: one
    // 128-byte line per thread
    {
        const long long nlines = (a.wk_gf * (long long)sizeof(double) + 127) / 128;
        const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
        for (long long l = t; l < nlines; l += (long long)gridDim.x * blockDim.x)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char *>(a.gf) + 128 * l));
    }
    const int k = blockIdx.x * 8 + warp;
    if (k >= a.nseg) return;
    double ru, rv;
    const InterpLane il = interp_lane(a, k, lane);
    interp_sum<T, LdNc>(a, (const T *)a.fin, il, ru, rv);
    if (lane == 0 && il.pos >= 0) {
        a.rhs[2 * il.pos] = ru;
        a.rhs[2 * il.pos + 1] = rv;
    }
}

// (D D^T)(k,l): the delta is separable, so the node sum over the box overlap
// is (sum_i phx_k phx_l)(sum_j phy_k phy_l)
__device__ __forceinline__ double bval(const Marker &mk, const Marker &ml)
{
    const int ia = max(mk.i1, ml.i1), ib = min(mk.i2, ml.i2);
    const int ja = max(mk.j1, ml.j1), jb = min(mk.j2, ml.j2);
    if (ia > ib || ja > jb) return 0.0;
    double sx = 0.0, sy = 0.0;
    for (int i = ia; i <= ib; ++i) sx += mk.phx[i - mk.i1] * ml.phx[i - ml.i1];
    for (int j = ja; j <= jb; ++j) sy += mk.phy[j - mk.j1] * ml.phy[j - ml.j1];
    return sx * sy;
}

__device__ __forceinline__ bool box_overlap(int4 p, int4 q)
{
    return max(p.x, q.x) <= min(p.y, q.y) && max(p.z, q.z) <= min(p.w, q.w);
}

// the marker at position srt of the solve order, or null (and the kernel's
// status bit set) when the order holds an index outside the markers or the
// marker is not as make_marker leaves it
__device__ __forceinline__ const Marker *sorted_marker(const IBArgs &a, int srt, unsigned bit)
{
    const int k = a.perm[srt];
    if (k < 0 || k >= a.nseg || !marker_ok(a, a.mk[k])) {
        atomicOr(a.status, bit);
        return nullptr;
    }
    return a.mk + k;
}

// Several bodies: sort the markers along the longer axis of the marker cloud
// (stable, ties by index) into perm/key, with reach = 6 lattice units along
// that axis. One CTA; dynamic shared memory key[ns] (double) + idx[ns] (int).
template <bool BATCH>
__global__ void __launch_bounds__(1024) ib_order(const IBArgs base0, const IBArgs *batch, int step0)
{
    const IBArgs &base = BATCH ? batch[blockIdx.z] : base0;
    const int step_index = factor_step<BATCH>(base, step0);
    if (step_index < 0) return;
    const IBArgs a = member_args(base, step_index);
    if (a.static_order) return;   // one rigid body: fixed order (batched launches reach it)
    extern __shared__ double osm[];
    const int n = a.nseg, tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;
    int ns = 1;
    while (ns < n) ns <<= 1;
    double *key = osm;
    int *idx = (int *)(key + ns);
    __shared__ double wext[32][4];
    __shared__ bool by_x;
    double lx0 = 1e300, lx1 = -1e300, ly0 = 1e300, ly1 = -1e300;
    for (int k = tid; k < n; k += nt) {
        const double xm = a.mk[k].xm, ym = a.mk[k].ym;
        lx0 = fmin(lx0, xm); lx1 = fmax(lx1, xm); ly0 = fmin(ly0, ym); ly1 = fmax(ly1, ym);
    }
    for (int off = 16; off; off >>= 1) {
        lx0 = fmin(lx0, __shfl_xor_sync(0xffffffffu, lx0, off));
        lx1 = fmax(lx1, __shfl_xor_sync(0xffffffffu, lx1, off));
        ly0 = fmin(ly0, __shfl_xor_sync(0xffffffffu, ly0, off));
        ly1 = fmax(ly1, __shfl_xor_sync(0xffffffffu, ly1, off));
    }
    if (lane == 0) { wext[warp][0] = lx0; wext[warp][1] = lx1; wext[warp][2] = ly0; wext[warp][3] = ly1; }
    __syncthreads();
    if (tid == 0) {
        double e0 = 1e300, e1 = -1e300, e2 = 1e300, e3 = -1e300;
        for (int w = 0; w < (nt >> 5); ++w) {
            e0 = fmin(e0, wext[w][0]); e1 = fmax(e1, wext[w][1]);
            e2 = fmin(e2, wext[w][2]); e3 = fmax(e3, wext[w][3]);
        }
        by_x = (e1 - e0) >= (e3 - e2);
        *a.reach = 6.0 * a.scale;
    }
    __syncthreads();
    for (int s2 = tid; s2 < ns; s2 += nt) {
        key[s2] = s2 < n ? (by_x ? a.mk[s2].xm : a.mk[s2].ym) : 1e300;
        idx[s2] = s2;
    }
    __syncthreads();
    for (int size = 2; size <= ns; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int s2 = tid; s2 < ns; s2 += nt) {
                const int t = s2 ^ stride;
                if (t > s2) {
                    const bool up = (s2 & size) == 0;
                    const bool gt = key[s2] > key[t] || (key[s2] == key[t] && idx[s2] > idx[t]);
                    if (gt == up) {
                        const double kk = key[s2]; key[s2] = key[t]; key[t] = kk;
                        const int ii = idx[s2]; idx[s2] = idx[t]; idx[t] = ii;
                    }
                }
            }
            __syncthreads();
        }
    for (int s2 = tid; s2 < n; s2 += nt) {
        a.perm[s2] = idx[s2];
        a.key[s2] = key[s2];
    }
}


// One CTA per block of BS markers in the solve order: the diagonal block D_b,
// the coupling L_b to block b-1, and the longest coupling in the order
// (half-bandwidth).
template <bool BATCH>
__global__ void __launch_bounds__(256) ib_assemble(const IBArgs base0, const IBArgs *batch, int step0)
{
    const IBArgs &base = BATCH ? batch[blockIdx.z] : base0;
    const int step_index = factor_step<BATCH>(base, step0);
    if (step_index < 0) return;
    const IBArgs a = member_args(base, step_index);
    const int n = a.nseg, blk = blockIdx.x, tid = threadIdx.x;
    if (blk >= (n + BS - 1) / BS) return;   // batched launches size the grid for the largest case
    __shared__ double ph[2 * BS][12];
    __shared__ int4 bx[2 * BS];
    __shared__ int wl;
    if (tid == 0) wl = 0;
    for (int q = tid; q < 2 * BS * 12; q += blockDim.x) {
        const int m = q / 12, c = q % 12, srt = (blk - 1) * BS + m;
        double v = 0.0;
        if (srt >= 0 && srt < n) {
            const Marker *mm = sorted_marker(a, srt, LBM_ST_INDEX_ASSEMBLE);
            if (mm) v = c < 6 ? mm->phx[c] : mm->phy[c - 6];
        }
        ph[m][c] = v;
    }
    for (int m = tid; m < 2 * BS; m += blockDim.x) {
        const int srt = (blk - 1) * BS + m;
        const Marker *mm = (srt >= 0 && srt < n) ? sorted_marker(a, srt, LBM_ST_INDEX_ASSEMBLE) : nullptr;
        bx[m] = mm ? mbox(*mm) : make_int4(1, 0, 1, 0);
        if (mm && m >= BS) a.mk[mm - a.mk].pos = srt;
    }
    __syncthreads();
    for (int q = tid; q < 2 * BS * BS; q += blockDim.x) {
        const bool lower = q >= BS * BS;
        const int r = (q % (BS * BS)) / BS, c = q % BS;
        const int mr = BS + r, mc = lower ? c : BS + c, sr = blk * BS + r;
        double v = 0.0;
        if (sr >= n) {
            v = (!lower && r == c) ? 1.0 : 0.0;
        } else if ((!lower && blk * BS + c < n) || (lower && blk > 0)) {
            const int4 p = bx[mr], o = bx[mc];
            const int ia = max(p.x, o.x), ib = min(p.y, o.y), ja = max(p.z, o.z), jb = min(p.w, o.w);
            if (ia <= ib && ja <= jb) {
                double sx = 0.0, sy = 0.0;
                for (int i = ia; i <= ib; ++i) sx += ph[mr][i - p.x] * ph[mc][i - o.x];
                for (int j = ja; j <= jb; ++j) sy += ph[mr][6 + j - p.z] * ph[mc][6 + j - o.z];
                v = sx * sy;
            }
        }
        const long long g = (long long)blk * BS * BS + r * BS + c;
        if (lower) a.bL[g] = v;
        else a.bD[g] = v;
    }
    // half-bandwidth: boxes (<= 6 nodes wide) overlap only for markers closer
    // than `reach` along the order's key (ascending in the solve order, so
    // the markers within reach are a run after srt). 16 threads per marker
    // of the block scan that run, thread l the markers srt + 1 + l + 16 i.
    {
        static_assert(BS * 16 == 256, "16 threads per marker of a block");
        const int m = tid >> 4, l = tid & 15, srt = blk * BS + m;
        if (srt < n) {
            const double reach = *a.reach;
            const int4 p = bx[BS + m];
            const double ks = a.key[srt];
            int w = 0;
            for (int t = srt + 1 + l; t < n && a.key[t] - ks <= reach; t += 16) {
                const Marker *mt = sorted_marker(a, t, LBM_ST_INDEX_ASSEMBLE);
                if (mt && box_overlap(p, mbox(*mt))) w = t - srt;
            }
            if (w) atomicMax(&wl, w);
        }
    }
    __syncthreads();
    if (tid == 0 && wl) atomicMax(a.wmax, wl);
}

// In-place inverse of one symmetric positive definite BS x BS block by one
// warp (Gauss-Jordan without pivoting, stable for SPD), row stride GP in
// shared memory. The block is held in registers during the BS elimination
// steps: lane (j, h) owns column j of rows 2e+h; the pivot row and column are
// broadcast by warp shuffles. Returns false if a pivot is not positive.
__device__ bool warp_inv(double *G)
{
    const int lane = threadIdx.x & 31;
    const int j = lane % BS, ih = lane / BS;
    double g[BS / 2];
#pragma unroll
    for (int e = 0; e < BS / 2; ++e) g[e] = G[(2 * e + ih) * GP + j];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < BS; ++k) {
        const int kh = k & 1, ke = k >> 1;            // owner half and register of row k
        const double p = __shfl_sync(0xffffffffu, g[ke], kh * BS + k);
        const bool good = p > 0.0 && isfinite(p);
        ok = ok && good;
        const double piv = good ? 1.0 / p : 1.0;
        const double rowk = __shfl_sync(0xffffffffu, g[ke], kh * BS + j) * piv;   // scaled G[k][j]
        double cik[BS / 2];
#pragma unroll
        for (int e = 0; e < BS / 2; ++e) cik[e] = __shfl_sync(0xffffffffu, g[e], ih * BS + k);   // G[2e+ih][k]
#pragma unroll
        for (int e = 0; e < BS / 2; ++e) {
            const int i = 2 * e + ih;
            if (i == k) g[e] = (j == k) ? piv : rowk;         // row k
            else if (j == k) g[e] = -cik[e] * piv;            // column k
            else g[e] = g[e] - cik[e] * rowk;                 // rank-1 update
        }
    }
#pragma unroll
    for (int e = 0; e < BS / 2; ++e) G[(2 * e + ih) * GP + j] = g[e];
    __syncwarp();
    return ok;
}

// n doubles (a multiple of 32) from global to shared memory, all loads in flight
template <int N>
__device__ __forceinline__ void stage(double *dst, const double *__restrict__ src)
{
    const int lane = threadIdx.x & 31;
    double v[N / 32];
#pragma unroll
    for (int it = 0; it < N / 32; ++it) v[it] = src[lane + 32 * it];
#pragma unroll
    for (int it = 0; it < N / 32; ++it) dst[lane + 32 * it] = v[it];
}

// BS x BS row-major block from global memory into the padded (GP) layout
__device__ __forceinline__ void stage_sq(double *dst, const double *__restrict__ src)
{
    const int lane = threadIdx.x & 31;
    double v[BS * BS / 32];
#pragma unroll
    for (int it = 0; it < BS * BS / 32; ++it) v[it] = src[lane + 32 * it];
#pragma unroll
    for (int it = 0; it < BS * BS / 32; ++it) {
        const int e = lane + 32 * it;
        dst[(e / BS) * GP + e % BS] = v[it];
    }
}


// Block products of the cyclic reduction. Lane 2r+h of a warp owns output
// row r (0..BS-1) and half h of the columns; B rows are read as 16-byte pairs
// that the two lanes of a row share, so a product costs BS x (1 + NH/2)
// shared loads per lane instead of two per multiply-add.
// acc[c] = sum_t A(r,t) B[t*ldb + h*NH + c], c < NH; A(r,t) is A[r][t] in the
// padded (GP) layout, or A[t][r] when TA.
template <int NH, bool TA>
__device__ __forceinline__ void rowmm(const double *A, const double *B, int ldb, double acc[NH])
{
    const int lane = threadIdx.x & 31, r = lane >> 1, h = lane & 1;
#pragma unroll
    for (int c = 0; c < NH; ++c) acc[c] = 0.0;
#pragma unroll
    for (int t = 0; t < BS; ++t) {
        const double a = TA ? A[t * GP + r] : A[r * GP + t];
        const double2 *b = reinterpret_cast<const double2 *>(B + t * ldb + h * NH);
#pragma unroll
        for (int c = 0; c < NH / 2; ++c) {
            const double2 bb = b[c];
            acc[2 * c] += a * bb.x;
            acc[2 * c + 1] += a * bb.y;
        }
    }
}

// dense fallback, factor: Cholesky L L^T of the full D D^T in the solve order
// (row-major, lower triangle, in place), whole CTA
__device__ void dense_factor(const IBArgs &a, int *bad)
{
    const int n = a.nseg, tid = threadIdx.x, nt = blockDim.x;
    const int warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
    double *L = a.B;
    for (long long q = tid; q < (long long)n * n; q += nt) {
        const int k = (int)(q / n), l = (int)(q % n);
        const Marker *mk = sorted_marker(a, k, LBM_ST_INDEX_FACTOR), *ml = sorted_marker(a, l, LBM_ST_INDEX_FACTOR);
        L[q] = mk && ml ? bval(*mk, *ml) : (k == l ? 1.0 : 0.0);
    }
    __syncthreads();
    for (int k = 0; k < n; ++k) {
        if (tid == 0) {
            const double d = L[(long long)k * n + k];
            double dk = 1.0;
            if (!(d > 0.0) || !isfinite(d)) *bad = 1;
            else dk = sqrt(d);
            L[(long long)k * n + k] = dk;
        }
        __syncthreads();
        const double dk = L[(long long)k * n + k];
        for (int i = k + 1 + tid; i < n; i += nt) L[(long long)i * n + k] /= dk;
        __syncthreads();
        for (int i = k + 1 + warp; i < n; i += nw) {
            const double lik = L[(long long)i * n + k];
            for (int j = k + 1 + lane; j <= i; j += 32) L[(long long)i * n + j] -= lik * L[(long long)j * n + k];
        }
        __syncthreads();
    }
}

// Factorization of one step's D D^T, one CTA of FACTOR_THREADS threads;
// dynamic shared memory: one block-operation workspace of WS doubles per warp.
// Block cyclic reduction: at stride st the active blocks are the multiples
// of st, and the odd multiples o are eliminated into their even neighbours.
// For each eliminated block the factor buffer keeps, row by row, BS x GW
// values [D_o^-1 | F_L | F_U] with F_L = D_o^-1 L_o (coupling to o - st) and
// F_U = D_o^-1 L_q^T (coupling to q = o + st); block 0, the last one left,
// keeps D_0^-1. The even neighbours are updated as
//   D_e -= L_q^T F_L(q) + L_e F_U(p),   L_e <- -L_e F_L(p)   (p = e - st, q = e + st).
template <bool BATCH>
__global__ void __launch_bounds__(FACTOR_THREADS, 65536 / (FACTOR_THREADS * 128)) ib_factor(const IBArgs base0, const IBArgs *batch, int step0)
{
    const IBArgs &base = BATCH ? batch[blockIdx.z] : base0;
    const int step_index = factor_step<BATCH>(base, step0);
    if (step_index < 0) return;
    const IBArgs a = member_args(base, step_index);
    extern __shared__ __align__(16) double Wbase[];
    const int n = a.nseg, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    __shared__ int bad, dense;
    __shared__ int bb[4];
    if (tid == 0) { bb[0] = 1 << 30; bb[1] = 1 << 30; bb[2] = -1; bb[3] = -1; }
    __syncthreads();
    // patch rectangle of the step: bounding box of all support boxes
    {
        int b0 = 1 << 30, b1 = 1 << 30, b2 = -1, b3 = -1;
        for (int k = tid; k < n; k += blockDim.x) {
            const int4 q = mbox(a.mk[k]);
            if (!box_in_bounds(q.x, q.y, q.z, q.w, a.nx, a.ny)) {
                atomicOr(a.status, LBM_ST_INDEX_FACTOR);
                continue;
            }
            if (q.y >= q.x && q.w >= q.z) { b0 = min(b0, q.x); b1 = min(b1, q.z); b2 = max(b2, q.y); b3 = max(b3, q.w); }
        }
        for (int off = 16; off; off >>= 1) {
            b0 = min(b0, __shfl_xor_sync(0xffffffffu, b0, off));
            b1 = min(b1, __shfl_xor_sync(0xffffffffu, b1, off));
            b2 = max(b2, __shfl_xor_sync(0xffffffffu, b2, off));
            b3 = max(b3, __shfl_xor_sync(0xffffffffu, b3, off));
        }
        if (lane == 0) { atomicMin(&bb[0], b0); atomicMin(&bb[1], b1); atomicMax(&bb[2], b2); atomicMax(&bb[3], b3); }
    }
    for (long long t = tid; t < a.st_tiles / (TILE_CAP + 1); t += blockDim.x)
        a.tiles[t * (TILE_CAP + 1)] = 0;   // tile counts, for ib_tile_scatter
    __syncthreads();
    if (tid == 0) {
        PatchInfo pi{0, 0, 0, 0};
        if (bb[2] >= bb[0]) {
            pi.i0 = bb[0]; pi.j0 = bb[1]; pi.w = bb[2] - bb[0] + 1; pi.h = bb[3] - bb[1] + 1;
            if (pi.w > a.patch_wmax || pi.h > a.patch_hmax) {
                atomicOr(a.status, LBM_ST_OVERFLOW);
                pi = PatchInfo{0, 0, 0, 0};
            }
        }
        *a.pinfo = pi;
        *a.nsup = 0;   // counted by ib_tile_scatter
        const int w = *a.wmax;
        bad = 0;
        dense = (w > BS || a.force_dense) ? 1 : 0;
        if (dense && !a.B) {   // ensure_ib rules this out
            atomicOr(a.status, LBM_ST_INDEX_FACTOR);
            dense = 0;
        }
        a.fmode[0] = dense;
        a.fmode[1] = w;
        *a.wmax = 0;   // for the next assembly
    }
    __syncthreads();
    if (n == 0) return;
    if (dense) {
        dense_factor(a, &bad);
        __syncthreads();
        if (tid == 0 && bad) atomicOr(a.status, LBM_ST_SOLVER);
        return;
    }
    const int nb = (n + BS - 1) / BS;
    double *Db = a.bD, *Lb = a.bL, *Gf = a.gf;
    double *W = Wbase + (long long)warp * WS;
    const int pr = lane >> 1, ph = lane & 1;   // product lane layout: row, column half
    for (int st = 1; st < nb; st <<= 1) {
        const int nodd = (nb - st + 2 * st - 1) / (2 * st);
        for (int m = warp; m < nodd; m += BOPS_WARPS) {
            const int o = st * (2 * m + 1), q2 = o + st;
            double *Gs = W, *Rs = W + BS * GP;   // D_o, then [L_o | L_q^T]
            stage_sq(Gs, Db + (long long)o * BS * BS);
            {
                double lv[BS * BS / 32], lq[BS * BS / 32];
#pragma unroll
                for (int it = 0; it < BS * BS / 32; ++it) {
                    lv[it] = Lb[(long long)o * BS * BS + lane + 32 * it];
                    lq[it] = q2 < nb ? Lb[(long long)q2 * BS * BS + lane + 32 * it] : 0.0;
                }
#pragma unroll
                for (int it = 0; it < BS * BS / 32; ++it) {
                    const int e = lane + 32 * it, r = e / BS, c = e % BS;
                    Rs[r * FL + c] = lv[it];
                    Rs[c * FL + BS + r] = lq[it];
                }
            }
            __syncwarp();
            if (!warp_inv(Gs) && lane == 0) bad = 1;
            double *Go = Gf + (long long)o * BS * GW + pr * GW;
#pragma unroll
            for (int c = 0; c < BS / 2; ++c) Go[ph * (BS / 2) + c] = Gs[pr * GP + ph * (BS / 2) + c];
            double acc[BS];
            rowmm<BS, false>(Gs, Rs, FL, acc);
            double2 *F2 = reinterpret_cast<double2 *>(Go + BS + ph * BS);
#pragma unroll
            for (int c = 0; c < BS / 2; ++c) F2[c] = make_double2(acc[2 * c], acc[2 * c + 1]);
            __syncwarp();
        }
        __syncthreads();
        const int neven = (nb + 2 * st - 1) / (2 * st);
        for (int m = warp; m < neven; m += BOPS_WARPS) {
            const int e = 2 * st * m, o1 = e - st, o2 = e + st;
            double *As = W, *Fs = W + BS * GP, *Ds = Fs + BS * FL;
            double *De = Db + (long long)e * BS * BS, *Le = Lb + (long long)e * BS * BS;
            stage_sq(Ds, De);
            if (o2 < nb) {   // D_e -= L_q^T F_L(q)
                stage_sq(As, Lb + (long long)o2 * BS * BS);
                const double *G = Gf + (long long)o2 * BS * GW + BS;
                double v[BS * BS / 32];
#pragma unroll
                for (int it = 0; it < BS * BS / 32; ++it) {
                    const int q = lane + 32 * it;
                    v[it] = G[(q / BS) * GW + q % BS];
                }
#pragma unroll
                for (int it = 0; it < BS * BS / 32; ++it) {
                    const int q = lane + 32 * it;
                    Fs[(q / BS) * FL + q % BS] = v[it];
                }
                __syncwarp();
                double acc[BS / 2];
                rowmm<BS / 2, true>(As, Fs, FL, acc);
#pragma unroll
                for (int c = 0; c < BS / 2; ++c) Ds[pr * GP + ph * (BS / 2) + c] -= acc[c];
                __syncwarp();
            }
            if (m > 0) {   // D_e -= L_e F_U(p), L_e <- -L_e F_L(p); lanes h = 0 hold the new L_e row
                stage_sq(As, Le);
                const double *G = Gf + (long long)o1 * BS * GW + BS;
                double v[BS * FL / 32];
#pragma unroll
                for (int it = 0; it < BS * FL / 32; ++it) {
                    const int q = lane + 32 * it;
                    v[it] = G[(q / FL) * GW + q % FL];
                }
#pragma unroll
                for (int it = 0; it < BS * FL / 32; ++it) Fs[lane + 32 * it] = v[it];
                __syncwarp();
                double acc[BS];
                rowmm<BS, false>(As, Fs, FL, acc);
                if (ph == 0) {
                    double2 *L2 = reinterpret_cast<double2 *>(Le + pr * BS);
#pragma unroll
                    for (int c = 0; c < BS / 2; ++c) L2[c] = make_double2(-acc[2 * c], -acc[2 * c + 1]);
                } else {
#pragma unroll
                    for (int c = 0; c < BS; ++c) Ds[pr * GP + c] -= acc[c];
                }
                __syncwarp();
            }
#pragma unroll
            for (int it = 0; it < BS * BS / 32; ++it) {
                const int q = lane + 32 * it;
                De[q] = Ds[(q / BS) * GP + q % BS];
            }
            __syncwarp();
        }
        __syncthreads();
    }
    // block 0: inverted by every warp on its own copy, stored by warp 0 (a
    // lone warp working while the others wait at the barrier was measured
    // several times slower)
    {
        double *Gs = W;
        stage_sq(Gs, Db);
        __syncwarp();
        const bool ok = warp_inv(Gs);
        if (warp == 0) {
            double *Go = Gf + pr * GW;
#pragma unroll
            for (int c = 0; c < BS / 2; ++c) Go[ph * (BS / 2) + c] = Gs[pr * GP + ph * (BS / 2) + c];
            if (!ok && lane == 0) bad = 1;
        }
    }
    __syncthreads();
    if (tid == 0 && bad) atomicOr(a.status, LBM_ST_SOLVER);
}

// The flow-dependent solve of one step, one CTA (solve_threads threads), with
// the cyclic-reduction factors of the step's slot:
//   forward, st = 1, 2, 4, ...:  r_e -= F_L(q)^T r_q + F_U(p)^T r_p  (even e)
//   block 0:                     x_0 = D_0^-1 r_0
//   backward, st = ..., 4, 2:    x_o = D_o^-1 r_o - F_L(o) x_p - F_U(o) x_q  (odd o)
// (F_L(q)^T = L_q^T D_q^-1 and F_U(p)^T = L_e D_p^-1 since D is symmetric.)
// The last backward level, half of the solution, is left to the tiles
// (marker_solution). What is left is a chain of log2(nb) levels each way in
// one SM, bound by latency: each level is a chain of 16 to 32 dependent
// multiply-adds and a barrier. So nothing else waits in it: the factor blocks
// of the levels from st0 on come into shared memory by bulk copies started
// before the right-hand sides are read, each warp has its first-level factors
// in registers by then, and 512 threads with 128 registers keep a level's
// operands in flight (1024 with 64: 1.2 us a level instead of 0.5).
// 1024 markers: 34 us -> 15 us alone. Also reports the errors of the
// factorization chain. Dynamic shared memory: the staged blocks, the
// right-hand sides (padded to whole blocks), the mbarrier.
template <bool BATCH>
__global__ void __launch_bounds__(SOLVE_THREADS, 1) ib_solve(const IBArgs a0, const IBArgs *batch)
{
    const IBArgs &a = BATCH ? batch[blockIdx.z] : a0;
    extern __shared__ __align__(128) double smem[];
    const int n = a.nseg, tid = threadIdx.x, nt = blockDim.x;
    const int warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
    const int nb = (n + BS - 1) / BS, st0 = solve_st0(nb), nres = (nb + st0 - 1) / st0;
    double *stage = smem, *X = smem + nres * BS * GW;
    uint64_t *bar = reinterpret_cast<uint64_t *>(X + 2 * nb * BS);
    if (BATCH) {   // a launch for several cases has room for each of them (launch_flow_batch_t)
        uint32_t have;
        asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(have));
        if (solve_bytes(nb, st0) > (int)have) {
            if (tid == 0) atomicOr(a.status, LBM_ST_INDEX_SOLVE);
            return;
        }
    }
    if (tid == 0) {
        mbar_init(bar, 1);
        mbar_init_fence();
    }
    __syncthreads();
    const bool dense = a.fmode[0] != 0;
    const double *Gf = a.gf;
    constexpr uint32_t kBlock = sizeof(double) * BS * GW;
    if (warp == 0 && !dense && n > 0) {
        if (lane == 0) mbar_expect_tx(bar, kBlock * (uint32_t)nres);
        __syncwarp();
        for (int m = lane; m < nres; m += 32)
            bulk_g2s(stage + m * BS * GW, Gf + (long long)m * st0 * BS * GW, kBlock, bar);
    }
    if (tid == nt - 1) {
        const unsigned fs = *a.fstatus;
        if (fs) { atomicOr(a.status, fs); *a.fstatus = 0u; }
        a.solve_res[1] = (double)a.fmode[1];
    }
    if (n == 0) return;
    if (dense) {
        for (int s = tid; s < n; s += nt) {
            X[s] = a.rhs[2 * s];
            X[n + s] = a.rhs[2 * s + 1];
        }
        __syncthreads();
        dense_tri(a, X, nt);
        __syncthreads();
        for (int s = tid; s < n; s += nt) {
            a.y[2 * s] = X[s];
            a.y[2 * s + 1] = X[n + s];
        }
        return;
    }
    // level 1: the warp's first even block's factors, then the right-hand sides
    const int i = lane & (BS - 1), c = lane >> 4;
    double fq[BS], fp[BS];
    const int e1 = 2 * warp;
    const bool q1 = e1 + 1 < nb, p1 = e1 > 0 && e1 < nb;
#pragma unroll
    for (int t = 0; t < BS; ++t) {
        fq[t] = q1 ? __ldg(Gf + ((long long)(e1 + 1) * BS + t) * GW + BS + i) : 0.0;
        fp[t] = p1 ? __ldg(Gf + ((long long)(e1 - 1) * BS + t) * GW + 2 * BS + i) : 0.0;
    }
    for (int s = tid; s < 2 * nb * BS; s += nt) X[s] = s < 2 * n ? a.rhs[s] : 0.0;
    __syncthreads();
    if (e1 < nb && nb > 1) {
        double acc = 0.0;
        if (q1) {
#pragma unroll
            for (int t = 0; t < BS; ++t) acc = rfma(fq[t], X[2 * ((e1 + 1) * BS + t) + c], acc);
        }
        if (p1) {
#pragma unroll
            for (int t = 0; t < BS; ++t) acc = rfma(fp[t], X[2 * ((e1 - 1) * BS + t) + c], acc);
        }
        X[2 * (e1 * BS + i) + c] -= acc;
    }
    for (int e = 2 * (warp + nw); e < nb; e += 2 * nw)
        bcr_forward(Gf + (long long)(e + 1) * BS * GW, Gf + (long long)(e - 1) * BS * GW, X, e, 1, e + 1 < nb, true, lane);
    // the staged blocks (bounded; copies that never land are reported, not
    // waited on forever)
    bool ok = true;
    int spins = 0;
    while (!mbar_try_wait(bar, 0))
        if (++spins > (1 << 22)) {
            ok = false;
            break;
        }
    if (__syncthreads_or(!ok)) {
        // wait (bounded) for copies still in flight before the CTA's shared
        // memory is released, and report
        if (tid == 0) atomicOr(a.status, LBM_ST_TIMEOUT);
        for (spins = 0; !mbar_try_wait(bar, 0) && spins < (1 << 22); ++spins) {
        }
        return;
    }
    auto block = [&](int o, int st) { return st >= st0 ? stage + o / st0 * BS * GW : Gf + (long long)o * BS * GW; };
    int st = 2;
    for (; st < nb; st <<= 1) {
        for (int e = 2 * st * warp; e < nb; e += 2 * st * nw) {
            const bool q = e + st < nb, p = e > 0;
            if (st >= st0)   // (two forms, so that staged reads are shared loads)
                bcr_forward(stage + (e + st) / st0 * BS * GW, stage + (e - st) / st0 * BS * GW, X, e, st, q, p, lane);
            else
                bcr_forward(block(e + st, st), block(e - st, st), X, e, st, q, p, lane);
        }
        __syncthreads();
    }
    if (warp == 0) bcr_root(stage, GW, X, lane);
    __syncthreads();
    for (st >>= 1; st > 1; st >>= 1) {
        for (int o = st * (2 * warp + 1); o < nb; o += 2 * st * nw) {
            if (st >= st0)
                bcr_backward(stage + o / st0 * BS * GW, X, o, st, o + st < nb, lane);
            else
                bcr_backward(block(o, st), X, o, st, o + st < nb, lane);
        }
        __syncthreads();
    }
    // the even blocks' solution (without a first level: all there is)
    for (int s = tid; s < 2 * n; s += nt)
        if ((s / (2 * BS) & 1) == 0) a.y[s] = X[s];
}

// Markers whose support box meets each 16 x 16 tile of the step's patch
// rectangle. Layout per tile: count, then up to TILE_CAP marker indices in
// increasing order (the order of the tile update's sums); a larger count
// tells the tile update to scan all markers for that tile. Geometry only, so
// part of the factorization chain, in two passes: each marker appends itself
// to the (at most 2 x 2) tiles its box meets, then each tile sorts its list.
// ib_factor has cleared the counts.
template <bool BATCH>
__global__ void __launch_bounds__(256) ib_tile_scatter(const IBArgs base0, const IBArgs *batch, int step0)
{
    const IBArgs &base = BATCH ? batch[blockIdx.z] : base0;
    const int step_index = factor_step<BATCH>(base, step0);
    if (step_index < 0) return;
    const IBArgs a = member_args(base, step_index);
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.nseg) return;
    const PatchInfo pi = *a.pinfo;
    const int4 q = mbox(a.mk[k]);
    if (!box_in_bounds(q.x, q.y, q.z, q.w, a.nx, a.ny)) {
        atomicOr(a.status, LBM_ST_INDEX_SCATTER);
        return;
    }
    if (q.y < q.x || q.w < q.z || pi.w <= 0) return;
    // the box lies in the patch rectangle (its bounding box), which the tile
    // grid covers; a box or rectangle that says otherwise is not indexed
    if (q.x < pi.i0 || q.z < pi.j0 || q.y >= pi.i0 + a.tiles_x * TILE ||
        (long long)((q.w - pi.j0) / TILE + 1) * a.tiles_x > patch_tiles(a)) {
        atomicOr(a.status, LBM_ST_INDEX_SCATTER);
        return;
    }
    const int tx0 = (q.x - pi.i0) / TILE, tx1 = (q.y - pi.i0) / TILE;
    const int ty0 = (q.z - pi.j0) / TILE, ty1 = (q.w - pi.j0) / TILE;
    for (int ty = ty0; ty <= ty1; ++ty)
        for (int tx = tx0; tx <= tx1; ++tx) {
            const int tile = ty * a.tiles_x + tx;
            int *list = a.tiles + (long long)tile * (TILE_CAP + 1);
            const int pos = atomicAdd(list, 1);
            if (pos < TILE_CAP) list[1 + pos] = k;
        }
}

// The step's correction tiles (those listing a marker) in ascending tile
// order, by a block scan of the tile counts: one CTA per member. The order
// fixes the order of the force sum, so the force rows do not depend on the
// order the scatter's atomics happened to run in.
template <bool BATCH>
__global__ void __launch_bounds__(256) ib_tile_compact(const IBArgs base0, const IBArgs *batch, int step0)
{
    const IBArgs &base = BATCH ? batch[blockIdx.z] : base0;
    const int step_index = factor_step<BATCH>(base, step0);
    if (step_index < 0) return;
    const IBArgs a = member_args(base, step_index);
    __shared__ int wsum[8];
    const int nt = (int)(a.st_tiles / (TILE_CAP + 1));
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int per = (nt + 255) / 256, b0 = min(nt, t * per), b1 = min(nt, b0 + per);
    int cnt = 0;
    for (int b = b0; b < b1; ++b) cnt += a.tiles[(long long)b * (TILE_CAP + 1)] > 0;
    int x = cnt;   // inclusive scan within the warp
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; ++w) before += wsum[w];
    int pos = before + x - cnt;
    for (int b = b0; b < b1; ++b)
        if (a.tiles[(long long)b * (TILE_CAP + 1)] > 0) a.ctile[pos++] = b;
    if (t == 255) *a.nsup = before + x;
}

// One warp per correction tile (8 per CTA): most tiles list a few dozen
// markers, which a warp sorts as fast as a CTA while holding an eighth of the
// SM slots the lattice update runs in.
constexpr int SORT_WARPS = 8;
// CTAs per step: 256 warps, about the correction tiles of a 1024-marker
// contour; larger contours loop
constexpr int SORT_CTAS = 32;
template <bool BATCH>
__global__ void __launch_bounds__(32 * SORT_WARPS) ib_tile_sort(const IBArgs base0, const IBArgs *batch, int step0)
{
    const IBArgs &base = BATCH ? batch[blockIdx.z] : base0;
    const int step_index = factor_step<BATCH>(base, step0);
    if (step_index < 0) return;
    const IBArgs a = member_args(base, step_index);
    __shared__ int keys[SORT_WARPS][TILE_CAP];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int *key = keys[warp];
    const int nt = patch_tiles(a);
    int ntile = *a.nsup;
    if (ntile < 0 || ntile > nt) {
        if (lane == 0) atomicOr(a.status, LBM_ST_INDEX_SORT);
        ntile = 0;
    }
    for (int c = blockIdx.x * SORT_WARPS + warp; c < ntile; c += gridDim.x * SORT_WARPS) {
        const int tile = a.ctile[c];
        if (tile < 0 || tile >= nt) {
            if (lane == 0) atomicOr(a.status, LBM_ST_INDEX_SORT);
            continue;
        }
        int *list = a.tiles + (long long)tile * (TILE_CAP + 1);
        const int m = min(list[0], TILE_CAP);
        int np = 2;   // keys sorted: the power of two at or above the count
        while (np < m) np <<= 1;
        for (int t = lane; t < np; t += 32) key[t] = t < m ? list[1 + t] : 0x7fffffff;
        __syncwarp();
        // bitonic sort of np keys, ascending (the padding keys stay at the
        // end); the pairs (t, t ^ stride) of a stage are disjoint
        for (int size = 2; size <= np; size <<= 1)
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int t = lane; t < np; t += 32) {
                    const int u = t ^ stride;
                    if (u > t) {
                        const bool up = (t & size) == 0;
                        const int x = key[t], y = key[u];
                        if ((x > y) == up) { key[t] = y; key[u] = x; }
                    }
                }
                __syncwarp();
            }
        for (int t = lane; t < m; t += 32) list[1 + t] = key[t];
        __syncwarp();
    }
}

// The step's force row from the correction tiles' partials, summed over the
// compact tile list in ascending tile order (deterministic), one CTA; no
// correction tile gives zero forces (solution.f90:327-330 normalisation).
// Needed by no kernel of the step, so it runs after the step's update.
__device__ __forceinline__ void force_row(const IBArgs &a, int rr)
{
    if (threadIdx.x == 32 && rr >= 0 && rr < a.ring_rows) {
        double time;
        const double *row = motion_row(a, a.cur_step, &time);
        write_header(a, row, time, rr);
    }
    __shared__ double red[8][NPART];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nt = patch_tiles(a);
    int ntile = a.nseg > 0 ? *a.nsup : 0;
    if (ntile < 0 || ntile > nt) {
        if (threadIdx.x == 0) atomicOr(a.status, LBM_ST_INDEX_FORCES);
        ntile = 0;
    }
    for (int w = 0; w < a.nwing; ++w) {
        double s0 = 0, s1 = 0, s2 = 0;
        for (int c = threadIdx.x; c < ntile; c += blockDim.x) {
            const int tile = a.ctile[c];
            if (tile < 0 || tile >= nt) {
                atomicOr(a.status, LBM_ST_INDEX_FORCES);
                continue;
            }
            const double *p = a.partial + (long long)tile * NPART + 3 * w;
            s0 += p[0]; s1 += p[1]; s2 += p[2];
        }
#pragma unroll
        for (int off = 16; off; off >>= 1) {
            s0 += __shfl_down_sync(0xffffffffu, s0, off);
            s1 += __shfl_down_sync(0xffffffffu, s1, off);
            s2 += __shfl_down_sync(0xffffffffu, s2, off);
        }
        if (lane == 0) { red[warp][3 * w] = s0; red[warp][3 * w + 1] = s1; red[warp][3 * w + 2] = s2; }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (rr < 0 || rr >= a.ring_rows) {
            atomicOr(a.status, LBM_ST_INDEX_FORCES);
            return;
        }
        double *fr = a.force_ring + (long long)rr * a.row_len;
        double tot[3] = {0, 0, 0};
        const double uu = a.uu, scale = a.scale;
        for (int w = 0; w < a.nwing; ++w) {
            double s0 = 0, s1 = 0, s2 = 0;
            for (int w8 = 0; w8 < 8; ++w8) { s0 += red[w8][3 * w]; s1 += red[w8][3 * w + 1]; s2 += red[w8][3 * w + 2]; }
            const double cx = 2.0 * s0 / (uu * uu * (1.0 / scale));
            const double cy = 2.0 * s1 / (uu * uu * (1.0 / scale));
            const double cm = -2.0 * s2 / (uu * uu * (1.0 / (scale * scale)));
            fr[1 + 3 * w] = cx; fr[2 + 3 * w] = cy; fr[3 + 3 * w] = cm;
            tot[0] += cx; tot[1] += cy; tot[2] += cm;
            if (!isfinite(cx) || !isfinite(cy) || !isfinite(cm)) atomicOr(a.status, LBM_ST_NONFINITE);
        }
        fr[1 + 3 * a.nwing] = tot[0];
        fr[2 + 3 * a.nwing] = tot[1];
        fr[3 + 3 * a.nwing] = tot[2];
    }
}

__global__ void __launch_bounds__(256) ib_forces(const IBArgs *batch)
{
    const IBArgs &a = batch[blockIdx.z];
    force_row(a, a.ring_row);
}

// arguments of case z of a batch's loop launch (they begin its entry)
__device__ __forceinline__ const IBArgs &loop_case(const void *batch, size_t stride)
{
    return *reinterpret_cast<const IBArgs *>((const char *)batch + blockIdx.z * stride);
}

// Residual of the step's solve, ||B y - rhs|| / ||rhs|| with B = D D^T
// recomputed from the marker geometry (independent of the factorization):
// one warp per row of the solve order, lanes over the couplings within the
// half-bandwidth; deterministic two-level sum (CTA partials, last CTA).
// Flags LBM_ST_SOLVER unless it is below 1e-6, or LBM_ST_NONFINITE when the
// right-hand side itself is not finite (the flow at the markers diverged).
// The sums go behind the slot's tile partials, the counter to their end.
__device__ __forceinline__ void solve_residual(const IBArgs &a, int blk)
{
    __shared__ double red[8][2];
    __shared__ bool amlast;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = a.nseg, s = blk * 8 + warp;
    const int nblk = (n + 7) / 8;
    double *partial = a.partial + (long long)NPART * patch_tiles(a);
    unsigned *counter = reinterpret_cast<unsigned *>(a.partial + a.st_part - 1);
    if (blk >= nblk) return;    // batched launches size the grid for the largest case
    const int hw = min(max((int)a.solve_res[1], 0), n);
    double rnum = 0.0, rden = 0.0;
    const int ks = s < n ? order_at(a, s, LBM_ST_INDEX_RESIDUAL) : -1;
    if (ks >= 0) {
        const Marker &ms = a.mk[ks];
        const bool ok_s = marker_ok(a, ms);
        if (!ok_s && lane == 0) atomicOr(a.status, LBM_ST_INDEX_RESIDUAL);
        double b0 = 0.0, b1 = 0.0;
        for (int t = s - hw + lane; t <= s + hw && ok_s; t += 32) {
            if (t < 0 || t >= n) continue;
            const Marker *ml = sorted_marker(a, t, LBM_ST_INDEX_RESIDUAL);
            if (!ml) continue;
            const double b = bval(ms, *ml);
            b0 += b * a.y[2 * t];
            b1 += b * a.y[2 * t + 1];
        }
#pragma unroll
        for (int off = 16; off; off >>= 1) {
            b0 += __shfl_xor_sync(0xffffffffu, b0, off);
            b1 += __shfl_xor_sync(0xffffffffu, b1, off);
        }
        const double q0 = a.rhs[2 * s], q1 = a.rhs[2 * s + 1];
        rnum = (b0 - q0) * (b0 - q0) + (b1 - q1) * (b1 - q1);
        rden = q0 * q0 + q1 * q1;
    }
    if (lane == 0) { red[warp][0] = rnum; red[warp][1] = rden; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t0 = 0, t1 = 0;
        for (int w = 0; w < 8; ++w) { t0 += red[w][0]; t1 += red[w][1]; }
        partial[2 * blk] = t0;
        partial[2 * blk + 1] = t1;
        __threadfence();
        amlast = atomicAdd(counter, 1u) == (unsigned)(nblk - 1);
    }
    __syncthreads();
    if (!amlast) return;
    __threadfence();
    double s0 = 0.0, s1 = 0.0;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
        s0 += __ldcg(partial + 2 * b);
        s1 += __ldcg(partial + 2 * b + 1);
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        s0 += __shfl_down_sync(0xffffffffu, s0, off);
        s1 += __shfl_down_sync(0xffffffffu, s1, off);
    }
    __syncthreads();
    if (lane == 0) { red[warp][0] = s0; red[warp][1] = s1; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double sn = 0, sd = 0;
        for (int w = 0; w < 8; ++w) { sn += red[w][0]; sd += red[w][1]; }
        const double res = sqrt(sn) / (sqrt(sd) + 1e-300);
        a.solve_res[0] = res;
        if (!isfinite(sd))
            atomicOr(a.status, LBM_ST_NONFINITE);
        else if (!(res < 1e-6))
            atomicOr(a.status, LBM_ST_SOLVER);
        *counter = 0u;
    }
}

__global__ void __launch_bounds__(256) ib_residual(const IBArgs *batch)
{
    const IBArgs &a = batch[blockIdx.z];
    if (!a.check_res) return;   // this case's step is not checked
    solve_residual(a, blockIdx.x);
}

// The force rows of `count` consecutive steps, headers included (CTA b: the
// step b after the arguments', of slot 0, into the row b after theirs), and the
// residual checks of the steps in `check` (bit t; `per` CTAs each), in one
// launch: they need nothing of one another, and a call of one step waits for
// both (us a call of one step, as kernels of their own and here: 400x200 48.5
// and 47, 1280x640 55 and 48). With BATCH the steps in `check` but not in `due`
// are the last ones of some cases (check_res).
template <bool BATCH>
__global__ void __launch_bounds__(256) ib_checks(const IBArgs a0, const void *batch, size_t stride, int count, unsigned check,
                                                 unsigned due, int per)
{
    const IBArgs &base = BATCH ? loop_case(batch, stride) : a0;
    const int b = blockIdx.x;
    if (b < count) {
        force_row(step_args(base, base.cur_step + b), base.ring_row + b);
        return;
    }
    const int q = (b - count) / per, blk = (b - count) - q * per;
    for (int k = 0; k < q; ++k) check &= check - 1;
    const int t = __ffs((int)check) - 1;
    if (t < 0 || t >= count || (BATCH && !((due >> t) & 1u) && !base.check_res)) return;
    solve_residual(step_args(base, base.cur_step + t), blk);
}

// The correction tiles of the step (the 16 x 16 tiles of the patch
// rectangle that list a marker), one CTA per tile: du = D^T y per node,
// gathered in marker order over the markers whose box covers the node (no
// atomics); then the lattice update of the tile's nodes with that velocity
// correction (the node path of the lattice kernels); and each node's FP64
// force and moment (boundary_condition.f90:1645-1675, solution.f90:327-336).
// Each tile's sums go to its partials, which the check after the step adds up
// (force_row). The lattice kernel updates every other node.
template <typename T, typename C, bool FIELDS, bool BATCH>
__global__ void __launch_bounds__(256) ib_tile_update(const IBArgs a0, const IBArgs *batch, const KFArgs<C> kf0,
                                                      const KFArgs<C> *kbatch, int step_index, int ring_slot)
{
    const IBArgs &a = BATCH ? batch[blockIdx.z] : a0;
    const KFArgs<C> &kf = BATCH ? kbatch[blockIdx.z] : kf0;
    __shared__ TileSmem S;
    __shared__ int smark[TILE_THREADS];   // the staged markers, where a list overflows
    const int nt = patch_tiles(a);
    const int ntile = *a.nsup;
    if (ntile == 0) return;   // no correction tile
    if (ntile < 0 || ntile > nt) {
        if (threadIdx.x == 0) atomicOr(a.status, LBM_ST_INDEX_TILE);
        return;
    }
    const PatchInfo pi = *a.pinfo;
    const T *__restrict__ fin = (const T *)kf.fin;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // the correction tiles, strided over the CTAs (the compact list is in no
    // particular order; each tile's result depends on the tile only)
    for (int c = blockIdx.x; c < ntile; c += gridDim.x) {
        const int tile = a.ctile[c];
        if (tile < 0 || tile >= nt) {   // the same for every thread of the CTA
            if (threadIdx.x == 0) atomicOr(a.status, LBM_ST_INDEX_TILE);
            continue;
        }
        const int ti0 = (tile % a.tiles_x) * TILE, tj0 = (tile / a.tiles_x) * TILE;
        const int *tlist = a.tiles + (long long)tile * (TILE_CAP + 1);
        const int listed = tlist[0];
        const int li = ti0 + tx, lj = tj0 + ty;                    // patch-relative
        const int gi = pi.i0 + li, gj = pi.j0 + lj;                // 0-based node
        bool active = li < pi.w && lj < pi.h;
        // the patch rectangle is the bounding box of the support boxes, all
        // interior nodes; a node outside the interior is not updated here
        if (active && (gi < 1 || gi > kf.nx - 2 || gj < 1 || gj > kf.ny - 2)) {
            atomicOr(a.status, LBM_ST_INDEX_TILE);
            active = false;
        }
        const int ta = pi.i0 + ti0, tb = ta + TILE - 1, sa_ = pi.j0 + tj0, sb_ = sa_ + TILE - 1;
        // the node's streamed populations first: their loads overlap the
        // staging of the markers
        C g[9];
        if (active) lbm_node::pull<T, C>(fin, kf.plane, kf.pitch, gi, gj, g);
        double du = 0.0, dv = 0.0;
        int wing = 1 << 20;
        if (listed <= TILE_CAP) {
            // markers listed for this tile by the factorization chain
            if ((int)threadIdx.x < listed) {
                const int k = tlist[1 + threadIdx.x];
                tile_stage(a, S, threadIdx.x, k);
            }
            tile_solve(a, S, listed, threadIdx.x, [&](int t) { return tlist[1 + t]; });
            __syncthreads();
            if (active) tile_gather(S, 0, listed, gi, gj, du, dv, wing);
        } else {
            // more markers than a list holds: scan all of them, in order
            for (int c0 = 0; c0 < a.nseg; c0 += 256) {
                const int k = c0 + threadIdx.x;
                bool hit = false;
                int4 q = make_int4(1, 0, 1, 0);
                if (k < a.nseg) {
                    if (marker_ok(a, a.mk[k])) {
                        q = mbox(a.mk[k]);
                        hit = q.x <= tb && q.y >= ta && q.z <= sb_ && q.w >= sa_ && q.y >= q.x;
                    } else {
                        atomicOr(a.status, LBM_ST_INDEX_TILE);
                    }
                }
                const unsigned bal = __ballot_sync(0xffffffffu, hit);
                if (lane == 0) S.wsum[warp] = __popc(bal);
                __syncthreads();
                if (threadIdx.x == 0) {
                    int acc = 0;
                    for (int w = 0; w < 8; ++w) { const int t = S.wsum[w]; S.wsum[w] = acc; acc += t; }
                    S.nlist = acc;
                }
                __syncthreads();
                if (hit) {
                    const int slot = S.wsum[warp] + __popc(bal & ((1u << lane) - 1u));
                    tile_stage(a, S, slot, k);
                    smark[slot] = k;
                }
                __syncthreads();
                tile_solve(a, S, S.nlist, threadIdx.x, [&](int t) { return smark[t]; });
                __syncthreads();
                if (active) tile_gather(S, 0, S.nlist, gi, gj, du, dv, wing);
                __syncthreads();
            }
        }
        // lattice update of the node with the correction, and its force and moment
        double fx = 0, fy = 0, mz = 0;
        const bool in_support = active && wing < (1 << 20);
        if (active) {
            C gout[9], frho, fu, fv;
            lbm_node::collide_interior<C>(kf, g, true, (C)du, (C)dv, gout, frho, fu, fv);
            lbm_node::store_node<T, C, FIELDS>(kf, (T *)kf.fout, gi, gj, gout, frho, fu, fv);
            if (in_support)
                node_force(a, motion_row(a, BATCH ? a.cur_step : step_index, nullptr), g, gi, gj, wing, du, dv, fx, fy, mz);
        }
        // deterministic tile reduction per wing, into the tile's partials
        tile_force_warp(a, S, in_support, wing, fx, fy, mz, warp, lane);
        __syncthreads();
        tile_force_store(a, S, tile, threadIdx.x);
        __syncthreads();   // shared arrays are reused by the next tile
    }
}


size_t order_smem(int n)
{
    int ns = 1;
    while (ns < n) ns <<= 1;
    return (sizeof(double) + sizeof(int)) * ns;
}

constexpr size_t kFactorSmem = sizeof(double) * BOPS_WARPS * WS;
constexpr size_t kSolveSmemMax = SOLVE_SMEM_BUDGET;
size_t solve_smem(int nseg)
{
    const int nb = (nseg + BS - 1) / BS;
    return (size_t)solve_bytes(nb, solve_st0(nb));
}

// Of a launch for several cases: the largest need among them, which is not
// that of the most markers (68 blocks keep every level above the first and
// take 226,320 bytes, 69 blocks every second one of those and 128,272).
size_t solve_smem(lbm_handle *const *hs, int n)
{
    size_t m = 0;
    for (int c = 0; c < n; ++c) m = std::max(m, solve_smem(hs[c]->nseg));
    return m;
}

// threads of the solve's CTA: one warp per even block of the first level
// (the widest), from 4 to SOLVE_THREADS / 32 warps. A solve of a few hundred
// markers then holds a fraction of an SM beside the lattice kernel instead
// of a whole one; each block's arithmetic is one warp's whatever the count,
// so the results do not depend on it.
int solve_threads(int nseg)
{
    const int nb = (nseg + BS - 1) / BS;
    return 32 * std::min(SOLVE_THREADS / 32, std::max(4, (nb + 1) / 2));
}

// arguments of the flow chain of the step held in buffer slot `slot`; for
// the batched factorization kernels, the arguments of slot 0 and member 0
// with the strides that member_args applies
IBArgs make_args(lbm_handle *h, const void *fin, int slot)
{
    const size_t ns = (size_t)(h->nseg > 0 ? h->nseg : 1);
    IBArgs a;
    a.fin = fin;
    a.prec = h->prec;
    a.nx = h->nx; a.ny = h->ny; a.pitch = h->pitch; a.plane = h->plane;
    a.nwing = h->nwing; a.ppw = h->ppw; a.spw = h->spw; a.nseg = h->nseg;
    a.smooth = h->p.delta_kernel;
    a.force_dense = (h->p.flags & LBM_FLAG_DENSE_SOLVE) != 0;
    a.scale = h->p.scale; a.ox = h->p.ox; a.oy = h->p.oy; a.uu = h->p.uu;
    a.xc = h->p.xc; a.yc = h->p.yc; a.mesh_max_scale = h->p.mesh_max_scale;
    a.xb0 = h->d_xb0; a.yb0 = h->d_yb0; a.arc = h->d_arc;
    a.mstep = h->d_mstep; a.msteps = h->msteps; a.mcols = h->mcols; a.mdt = h->mdt;
    a.nslots = h->nslots;
    a.static_order = h->static_order;
    a.st_mk = (long long)ns;
    a.st_perm = h->static_order ? 0 : (long long)ns;
    a.st_B = h->d_B ? (long long)(ns * ns) : 0;
    a.wk_blocks = (long long)h->work_blocks;
    a.wk_gf = (long long)h->gf_slot;
    a.mk = h->d_mk + slot * ns;
    a.perm = h->d_perm + slot * a.st_perm;
    a.key = h->d_key + slot * a.st_perm;
    a.B = h->d_B + slot * a.st_B;
    a.fmode = h->d_fmode + 2 * slot;
    a.fstatus = h->d_fstatus + slot;
    a.pinfo = h->d_pinfo + slot;
    a.tiles_x = h->patch_gx();
    a.st_tiles = (long long)h->patch_gx() * h->patch_gy() * (TILE_CAP + 1);
    a.tiles = h->d_tiles + slot * a.st_tiles;
    a.gf = h->d_gf + slot * h->gf_slot;
    // the step's own right-hand sides, solution, tile partials and residual,
    // one set per slot: the check of a step may run while later steps' flow
    // chains fill theirs
    a.st_rhs = 2ll * (long long)ns;
    a.st_part = (long long)h->part_stride;
    a.rhs = h->d_rhs + slot * a.st_rhs; a.y = h->d_y + slot * a.st_rhs;
    a.bD = h->d_bD; a.bL = h->d_bL;
    a.reach = h->d_reach; a.wmax = h->d_wmax;
    a.nsup = h->d_nsup + slot;
    a.ctile = h->d_ctile + slot * (a.st_tiles / (TILE_CAP + 1));
    a.patch_wmax = h->patch_wmax; a.patch_hmax = h->patch_hmax;
    a.partial = h->d_partial + slot * a.st_part;
    a.force_ring = h->d_ring; a.row_len = h->row_len;
    a.ring_row = 0; a.ring_rows = h->ring_cap;
    a.status = h->d_status; a.solve_res = h->d_solve_res + 2 * slot;
    a.cur_step = h->n;
    a.fstep0 = 0; a.fcount = 0;
    a.check_res = 1;
    return a;
}

template <typename T, typename C>
int launch_flow_t(lbm_handle *h, const void *fin, void *fout, void *fields, int step_index, int ring_slot, int slot,
                  cudaStream_t st, cudaEvent_t after_interp)
{
    IBArgs a = make_args(h, fin, slot);
    if (h->nseg > 0) {
        ib_interp<T, false><<<(h->nseg + 7) / 8, 256, 0, st>>>(a, nullptr);
        h->count(1);
    }
    if (after_interp && cudaEventRecord(after_interp, st) != cudaSuccess) return -1;
    ib_solve<false><<<1, solve_threads(h->nseg), solve_smem(h->nseg), st>>>(a, nullptr);
    const int grid = std::min(h->patch_gx() * h->patch_gy(), 2 * 148);   // strided over the correction tiles
    const KFArgs<C> kf = make_kf_args<C>(h, fin, fout, fields, KF_OUTER);
    if (fields)
        ib_tile_update<T, C, true, false><<<grid, 256, 0, st>>>(a, nullptr, kf, nullptr, step_index, ring_slot);
    else
        ib_tile_update<T, C, false, false><<<grid, 256, 0, st>>>(a, nullptr, kf, nullptr, step_index, ring_slot);
    h->count(2);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// the force rows of `count` steps from step0 on and the residual checks of
// those in `check`
int launch_checks(lbm_handle *h, int step0, int count, int ring_slot, unsigned check, cudaStream_t st)
{
    IBArgs a = make_args(h, nullptr, 0);
    a.cur_step = step0;
    a.ring_row = ring_slot;
    const int per = (h->nseg + 7) / 8, checks = per > 0 ? __builtin_popcount(check) : 0;
    ib_checks<false><<<count + checks * per, 256, 0, st>>>(a, nullptr, 0, count, check, check, std::max(per, 1));
    h->count(count + checks, 1);   // a force row of each step, a check
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace

// per-CTA partials of ib_tile_update (doubles)
int ib_partials_per_block() { return NPART; }

// ints per patch tile of the tile lists (count + TILE_CAP indices)
int ib_tile_ints() { return TILE_CAP + 1; }

// scratch of the block cyclic reduction (doubles): working diagonal and
// coupling blocks (one set), and the factor buffer of one slot
void ib_factor_scratch(int nseg, size_t *work_blocks, size_t *factor_slot)
{
    const size_t nb = (size_t)(nseg + BS - 1) / BS;
    *work_blocks = nb * BS * BS;
    *factor_slot = nb * BS * GW;
}

int ib_max_markers() { return NMARK_MAX; }

template <bool BATCH>
int ib_configure_t()
{
    if (cudaFuncSetAttribute(ib_factor<BATCH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFactorSmem) !=
        cudaSuccess)
        return -1;
    if (cudaFuncSetAttribute(ib_solve<BATCH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSolveSmemMax) !=
        cudaSuccess)
        return -1;
    if (cudaFuncSetAttribute(ib_order<BATCH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)order_smem(NMARK_MAX)) != cudaSuccess)
        return -1;
    return 0;
}

int ib_configure(lbm_handle *h)
{
    (void)h;
    return ib_configure_t<false>() || ib_configure_t<true>() ? -1 : 0;
}

// factorization chains of the `count` steps step0, step0+1, ... (each into
// its slot), one launch per kernel with the steps along grid y
int launch_factor(lbm_handle *h, int step0, int count, cudaStream_t st)
{
    if (h->nseg == 0 || count <= 0) return 0;
    const IBArgs a = make_args(h, nullptr, 0);
    const int nb = (h->nseg + BS - 1) / BS;
    ib_geometry<false><<<dim3((h->nseg + 127) / 128, count), 128, 0, st>>>(a, nullptr, step0);
    if (!h->static_order) ib_order<false><<<dim3(1, count), 1024, order_smem(h->nseg), st>>>(a, nullptr, step0);
    ib_assemble<false><<<dim3(nb, count), 256, 0, st>>>(a, nullptr, step0);
    ib_factor<false><<<dim3(1, count), FACTOR_THREADS, kFactorSmem, st>>>(a, nullptr, step0);
    ib_tile_scatter<false><<<dim3((h->nseg + 255) / 256, count), 256, 0, st>>>(a, nullptr, step0);
    ib_tile_compact<false><<<dim3(1, count), 256, 0, st>>>(a, nullptr, step0);
    const int sort_ctas = std::min((h->patch_gx() * h->patch_gy() + SORT_WARPS - 1) / SORT_WARPS, SORT_CTAS);
    ib_tile_sort<false><<<dim3(sort_ctas, count), 32 * SORT_WARPS, 0, st>>>(a, nullptr, step0);
    h->count(h->static_order ? 6 : 7);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_check_steps(lbm_handle *h, int step0, int count, int ring_slot, bool last, cudaStream_t st)
{
    unsigned check = 0;
    for (int t = 0; t < count; ++t)
        if (check_due(step0 + t) || (last && t == count - 1)) check |= 1u << t;
    return launch_checks(h, step0, count, ring_slot, check, st);
}

// force row and residual check of one step, after its flow chain
int launch_check(lbm_handle *h, int step, int ring_slot, bool residual, cudaStream_t st)
{
    return launch_checks(h, step, 1, ring_slot, residual ? 1u : 0u, st);
}

// flow chain of step `step_index`: interpolation, solve with the factor of
// `slot`, spread and forces
int launch_flow(lbm_handle *h, const void *fin, void *fout, void *fields, int step_index, int ring_slot, int slot,
                cudaStream_t st, cudaEvent_t after_interp)
{
    if (!st) st = h->stream;
    switch (h->prec) {
    case LBM_PREC_FP32:
        return launch_flow_t<float, float>(h, fin, fout, fields, step_index, ring_slot, slot, st, after_interp);
    case LBM_PREC_FP64:
        return launch_flow_t<double, double>(h, fin, fout, fields, step_index, ring_slot, slot, st, after_interp);
    case LBM_PREC_FP16:
        return launch_flow_t<__half, float>(h, fin, fout, fields, step_index, ring_slot, slot, st, after_interp);
    case LBM_PREC_BF16:
        return launch_flow_t<__nv_bfloat16, float>(h, fin, fout, fields, step_index, ring_slot, slot, st, after_interp);
    }
    return -1;
}

// ---- batches of cases (lbm_batch.cu): arguments from device arrays, one
// launch per kernel for all cases (grid z = case), grids sized for the
// largest case

size_t ib_args_size() { return sizeof(IBArgs); }

void ib_args_write(lbm_handle *h, const void *fin, int slot, void *dst) { *(IBArgs *)dst = make_args(h, fin, slot); }

void ib_factor_args_write(lbm_handle *h, int step0, int count, void *dst)
{
    IBArgs a = make_args(h, nullptr, 0);
    a.fstep0 = step0;
    a.fcount = count;
    *(IBArgs *)dst = a;
}

namespace {

int max_seg(lbm_handle *const *hs, int n)
{
    int m = 0;
    for (int c = 0; c < n; ++c) m = std::max(m, hs[c]->nseg);
    return m;
}

constexpr int kBatchTileCtas = 64;

template <typename T, typename C>
int launch_flow_batch_t(lbm_handle *const *hs, int ncase, const IBArgs *dargs, const void *dkf, int step_index,
                        int ring_slot, bool fields, cudaStream_t st, cudaEvent_t after_interp)
{
    const int ns = max_seg(hs, ncase);
    ib_interp<T, true><<<dim3((ns + 7) / 8, 1, ncase), 256, 0, st>>>(IBArgs{}, dargs);
    if (after_interp && cudaEventRecord(after_interp, st) != cudaSuccess) return -1;
    ib_solve<true><<<dim3(1, 1, ncase), solve_threads(ns), solve_smem(hs, ncase), st>>>(IBArgs{}, dargs);
    // CTAs per case, strided over the case's correction tiles: the patch
    // grids bound the tiles several times over (a sweep case of chord 256
    // has some 60 correction tiles in a grid of hundreds), and CTAs past a
    // case's tiles still take lattice slots at the flow chain's priority, so
    // a batch launches at most kBatchTileCtas per case
    int tiles = 1;
    for (int c = 0; c < ncase; ++c) tiles = std::max(tiles, hs[c]->patch_gx() * hs[c]->patch_gy());
    const dim3 grid(std::min(tiles, kBatchTileCtas), 1, ncase);
    const KFArgs<C> *kf = (const KFArgs<C> *)dkf;
    if (fields)
        ib_tile_update<T, C, true, true><<<grid, 256, 0, st>>>(IBArgs{}, dargs, KFArgs<C>{}, kf, step_index, ring_slot);
    else
        ib_tile_update<T, C, false, true><<<grid, 256, 0, st>>>(IBArgs{}, dargs, KFArgs<C>{}, kf, step_index, ring_slot);
    for (int c = 0; c < ncase; ++c) hs[c]->count(3);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace

// factorization chains of the steps step0 .. step0+count-1 of every case
int launch_factor_batch(lbm_handle *const *hs, int ncase, const void *dargs, int step0, int count, cudaStream_t st)
{
    if (ncase <= 0 || count <= 0) return 0;
    const IBArgs *d = (const IBArgs *)dargs;
    const int ns = max_seg(hs, ncase), nb = (ns + BS - 1) / BS;
    bool any_order = false;
    int tiles = 1;
    for (int c = 0; c < ncase; ++c) {
        any_order = any_order || !hs[c]->static_order;
        tiles = std::max(tiles, hs[c]->patch_gx() * hs[c]->patch_gy());
    }
    ib_geometry<true><<<dim3((ns + 127) / 128, count, ncase), 128, 0, st>>>(IBArgs{}, d, step0);
    if (any_order) ib_order<true><<<dim3(1, count, ncase), 1024, order_smem(ns), st>>>(IBArgs{}, d, step0);
    ib_assemble<true><<<dim3(nb, count, ncase), 256, 0, st>>>(IBArgs{}, d, step0);
    ib_factor<true><<<dim3(1, count, ncase), FACTOR_THREADS, kFactorSmem, st>>>(IBArgs{}, d, step0);
    ib_tile_scatter<true><<<dim3((ns + 255) / 256, count, ncase), 256, 0, st>>>(IBArgs{}, d, step0);
    ib_tile_compact<true><<<dim3(1, count, ncase), 256, 0, st>>>(IBArgs{}, d, step0);
    ib_tile_sort<true><<<dim3(std::min((tiles + SORT_WARPS - 1) / SORT_WARPS, SORT_CTAS), count, ncase),
                         32 * SORT_WARPS, 0, st>>>(IBArgs{}, d, step0);
    for (int c = 0; c < ncase; ++c) hs[c]->count(any_order ? 7 : 6);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// flow chains of one step of every case (dargs: the cases' arguments of the
// step's slot; dkf: their lattice arguments)
int launch_flow_batch(lbm_handle *const *hs, int ncase, const void *dargs, const void *dkf, int step_index,
                      int ring_slot, bool fields, cudaStream_t st, cudaEvent_t after_interp)
{
    if (ncase <= 0) return 0;
    const IBArgs *d = (const IBArgs *)dargs;
    switch (hs[0]->prec) {
    case LBM_PREC_FP32:
        return launch_flow_batch_t<float, float>(hs, ncase, d, dkf, step_index, ring_slot, fields, st, after_interp);
    case LBM_PREC_FP64:
        return launch_flow_batch_t<double, double>(hs, ncase, d, dkf, step_index, ring_slot, fields, st, after_interp);
    case LBM_PREC_FP16:
        return launch_flow_batch_t<__half, float>(hs, ncase, d, dkf, step_index, ring_slot, fields, st, after_interp);
    case LBM_PREC_BF16:
        return launch_flow_batch_t<__nv_bfloat16, float>(hs, ncase, d, dkf, step_index, ring_slot, fields, st,
                                                         after_interp);
    }
    return -1;
}

// force rows and residual checks of one step of every case
int launch_check_batch(lbm_handle *const *hs, int ncase, const void *dargs, int ring_slot, bool residual,
                       cudaStream_t st)
{
    if (ncase <= 0) return 0;
    const IBArgs *d = (const IBArgs *)dargs;
    const int ns = max_seg(hs, ncase);
    ib_forces<<<dim3(1, 1, ncase), 256, 0, st>>>(d);
    for (int c = 0; c < ncase; ++c) hs[c]->count(1);
    if (!residual) return cudaGetLastError() == cudaSuccess ? 0 : -1;   // no case checks this step
    ib_residual<<<dim3((ns + 7) / 8, 1, ncase), 256, 0, st>>>(d);
    for (int c = 0; c < ncase; ++c) hs[c]->count(1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_check_steps_batch(lbm_handle *const *hs, int ncase, const void *dargs, size_t stride, int count, unsigned due,
                             bool last, cudaStream_t st)
{
    const int ns = max_seg(hs, ncase);
    const unsigned check = due | (last ? 1u << (count - 1) : 0u);
    const int per = (ns + 7) / 8, checks = __builtin_popcount(check);
    ib_checks<true><<<dim3(count + checks * per, 1, ncase), 256, 0, st>>>(IBArgs{}, dargs, stride, count, check, due, per);
    for (int c = 0; c < ncase; ++c) hs[c]->count(count + checks, 1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
