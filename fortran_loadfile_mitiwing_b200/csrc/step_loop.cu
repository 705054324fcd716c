// step_loop.cu -- several time steps of a small case in one launch.
//
// On a lattice whose populations stay in L2 a step is not bound by memory but
// by the chain of its dependent stages: interpolation -> solve -> correction
// tiles -> next step. As separate launches each link costs a kernel's start
// and end and a cross-stream event besides its own arithmetic. Here one
// cooperative launch runs up to a factorization batch of steps, and its CTAs
// (one per SM) hand the stages to one another through L2:
//
//   CTA 0       the solver: stages the step's factor blocks in shared memory
//               while the markers are interpolated, solves as soon as the
//               right-hand sides are there, and publishes the solution
//   other CTAs  interpolation (a warp per marker); then, while the solver
//               works, every lattice node outside the correction tiles, and
//               the correction tiles' markers and populations brought on
//               chip; then, with the solution, the correction tiles; and a
//               barrier among themselves before the next step
//
// Right-hand sides and solutions are their own flags: the factorization chain
// leaves not_yet() in the step's slot and the reader polls the value it needs,
// which saves a fence, a counter and a second round trip per hand-over (with a
// counter each, a 96x64 step took 15.2 us). What the next stage needs besides
// (a marker's weights, the markers of a tile) is loaded a step ahead, off the
// chain, and what it does not need (the forces of a tile) is left for after.
//
// Measured on a B200, us a step, launches per stage -> here: 96x64 27.9 ->
// 8.1; 400x200 33.5 -> 9.3 (FP64 31.7 -> 10.9); 1001x501 with two wings
// 42 -> 13.2; 1280x640 42 -> 13.6; 2048x1024 in BF16 46 -> 25.4, of which
// 20 are the lattice (with its loads through registers 24).
// On large lattices the staged kernel is the better one (loop_fits).
//
// The force rows and residual checks of the steps follow as ordinary launches
// (what they read is kept per step slot). Populations, right-hand sides and
// solutions are read from L2 (LdCg): other CTAs wrote them in this launch.
// Every wait is bounded; one that gives up sets LBM_ST_TIMEOUT and a flag
// that ends the other CTAs' waits too.
#include <algorithm>
#include <type_traits>

#include "ib_device.cuh"

namespace {

using namespace lbm_ib;
using namespace lbm_node;

constexpr int LOOP_STEPS = LBM_NSLOT_MAX / 2;   // steps of one launch at most (a slot half)
// counters, each on a line of its own
enum { SYNC_STEP = 0, SYNC_ABORT = 32, SYNC_WORDS = 64 };
// dynamic shared memory a CTA may use: a block's 227 KB less the kernel's
// static part (up to 1536 bytes, for batches in FP64). The kernels' limit is
// set to it, the same for every handle: the attribute is the process's, and
// another thread may set it between this one's setting and its launch.
constexpr int LOOP_SMEM = 232448 - 1536;

// Shares of the interior items (measured on 1280x640, 131 CTAs of which some 24
// have a tile and each CTA some 97 items; us a step): items dealt out evenly
// 15.4; a CTA with a tile 24, 36, 48 less 14.6, 15.0, 15.1; besides, all items
// taken as the warps come 13.9, 13.5, 13.6; the last 2 or 4 a warp (36 less)
// 13.6, 14.1. On 2048x1024 in BF16 (248 items a CTA) taking all costs more
// than it saves: 25.3, 25.6 (24 less), 25.9 (all taken), 25.4 (the last 2).
constexpr int LEAN = 36, TAIL = 2;
constexpr int NT = 512;                         // threads of a CTA (at 1024 the 64 registers left to each spill)

template <typename C> struct LoopArgs {
    IBArgs ib;               // slot 0
    KFArgs<C> kf;            // fin, fout, tiles, pinfo and the field pointers are not used
    void *f[2];              // population buffers: step s reads f[s & 1], writes the other
    C *fields[LOOP_STEPS];   // rho, u, v of a step (nx*ny each), or null
    int step0, nsteps;
    unsigned *sync;          // SYNC_WORDS counters; base: what the step counter holds at the launch
    unsigned base;
};

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_release(unsigned *p, unsigned v)
{
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

constexpr int SPINS = 1 << 22;

// a wait of this CTA gave up: report it and end the other CTAs' waits
__device__ __forceinline__ void give_up(unsigned *sync, unsigned *status)
{
    atomicOr(status, LBM_ST_TIMEOUT);
    red_release(sync + SYNC_ABORT, 1u);
}

// bounded wait for the step counter to reach target (one thread); false when
// it gave up or another CTA did
__device__ __forceinline__ bool wait_step(unsigned *sync, unsigned target, unsigned *status)
{
    for (int spins = 0; spins < SPINS; ++spins) {
        if ((int)(ld_acquire(sync + SYNC_STEP) - target) >= 0) return true;
        if ((spins & 63) == 63 && ld_acquire(sync + SYNC_ABORT)) return false;
    }
    give_up(sync, status);
    return false;
}

// bounded wait for the two values p[0] and p[1] of a marker (right-hand sides
// or solution); false when it gave up or another CTA did
__device__ __forceinline__ bool wait_pair(const double *p, unsigned *sync, unsigned *status, double &x, double &y)
{
    for (int spins = 0; spins < SPINS; ++spins) {
        long long a, b;
        asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
        asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(b) : "l"(p + 1) : "memory");
        if (a != (long long)LBM_NOT_YET && b != (long long)LBM_NOT_YET) {
            x = __longlong_as_double(a);
            y = __longlong_as_double(b);
            return true;
        }
        if ((spins & 63) == 63 && ld_acquire(sync + SYNC_ABORT)) return false;
    }
    give_up(sync, status);
    return false;
}
__device__ __forceinline__ void put_value(double *p, double x)
{
    const long long v = __double_as_longlong(is_value(x));
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// shared memory of a tile's threads
struct GroupSmem {
    TileSmem tile;
    TileWeights weights;
};

__device__ __forceinline__ void group_sync(int grp)
{
    asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "r"(TILE_THREADS) : "memory");
}

template <typename C>
__device__ __forceinline__ void put_fields(C *fl, long long nn, long long q, C rho, C u, C v)
{
    fl[q] = rho;
    fl[nn + q] = u;
    fl[2 * nn + q] = v;
}

template <typename T, typename C>
__device__ __forceinline__ void put_node(const KFArgs<C> &a, T *fout, C *fl, int i, int j, const C gout[9], C rho, C u, C v)
{
    const long long o = (long long)j * a.pitch + i;
#pragma unroll
    for (int k = 0; k < 9; ++k) Store<T>::st(fout + (long long)k * a.plane + o, gout[k]);
    if (fl) put_fields(fl, (long long)a.nx * a.ny, (long long)j * a.nx + i, rho, u, v);
}

// node (i, j) lies in a correction tile of the step
__device__ __forceinline__ bool in_tile(const IBArgs &a, const PatchInfo &r, int i, int j)
{
    const unsigned li = (unsigned)(i - r.i0), lj = (unsigned)(j - r.j0);
    if (li >= (unsigned)r.w || lj >= (unsigned)r.h) return false;
    const unsigned tx = li >> 4, t = (lj >> 4) * (unsigned)a.tiles_x + tx;
    if (tx >= (unsigned)a.tiles_x || t >= (unsigned)patch_tiles(a)) {
        atomicOr(a.status, LBM_ST_INDEX_LATTICE);
        return false;
    }
    return a.tiles[(long long)t * (TILE_CAP + 1)] > 0;
}

// One warp's item of the interior: with FP32 arithmetic two nodes per lane
// (rows j, j + 1 of a column, or with 2-byte storage columns i, i + 1 of a
// row) by the paired update, as in the staged lattice kernel; one node per
// lane in FP64. An item's rows come into the warp's part of shared memory by
// 16-byte asynchronous copies (through L2: other CTAs wrote them), some items
// ahead: with loads into registers, of which 512 threads have 128 each, only
// one item's were in flight and a third of the time went into waiting for them.
template <typename T> struct Items {
    static constexpr int AL = 16 / (int)sizeof(T);                // elements of a copy
    static constexpr int COLS = sizeof(T) == 2 ? 64 : 32;         // of an item
    static constexpr int ROWS = sizeof(T) == 4 ? 2 : 1;
    static constexpr int SEG = COLS / AL;                         // copies of a row's segment, one more where it is shifted
    static constexpr int ROW = 9 * SEG + 6;                       // copies of a row
    static constexpr int BYTES = ROWS * ROW * 16;
    static constexpr int STAGES = sizeof(T) == 2 ? 4 : 2;
    // the first copy of population k's segment
    static __host__ __device__ constexpr int at(int k)
    {
        int c = 0;
        for (int q = 0; q < k; ++q) c += SEG + (lbm_ex(q) != 0);
        return c;
    }
};

// offsets of a row's copies from its node (i0, j), for the launch
template <typename T> __device__ __forceinline__ void item_table(int *tab, int plane, int pitch)
{
    using I = Items<T>;
    for (int c = threadIdx.x; c < I::ROW; c += NT) {
        int k = 0, q = c;
        while (q >= I::SEG + (lbm_ex(k) != 0)) {
            q -= I::SEG + (lbm_ex(k) != 0);
            ++k;
        }
        tab[c] = k * plane - lbm_ey(k) * pitch + (q - (lbm_ex(k) == 1)) * I::AL;   // (9 planes < 2^31 elements, loop_fits)
    }
}

// A warp's copies of an item into its stage. The segments' ends may lie up to
// 16 bytes outside the rows; the buffers are padded for that.
template <typename T, typename C>
__device__ __forceinline__ void item_issue(const KFArgs<C> &a, const T *fin, const int *tab, unsigned char *stage, int item,
                                           int segs, int lane)
{
    using I = Items<T>;
    const int r = item / segs, sg = item - r * segs, j = 1 + I::ROWS * r;
    const T *row = fin + j * a.pitch + sg * I::COLS;
    const int up = I::ROWS == 2 && j + 1 <= a.ny - 2 ? a.pitch : 0;   // an odd last row fills both halves
    const uint32_t dst = smem_u32(stage);
#pragma unroll
    for (int t = 0; t < (I::ROWS * I::ROW + 31) / 32; ++t) {
        const int c = 32 * t + lane;
        if (c < I::ROWS * I::ROW) {
            const bool second = I::ROWS == 2 && c >= I::ROW;
            const T *src = row + tab[second ? c - I::ROW : c] + (second ? up : 0);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * c), "l"(__cvta_generic_to_global(src)) : "memory");
        }
    }
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <typename T> struct LatticeItem {
    float2 g[9];
    int i, j;
    bool w0, w1;   // first, second node is written
};
template <> struct LatticeItem<double> {
    double g[9];
    int i, j;
    bool w0, w1;
};

template <typename T, typename C>
__device__ __forceinline__ void item_nodes(LatticeItem<T> &x, const KFArgs<C> &a, const IBArgs &ib, const PatchInfo &pr, int item,
                                           int segs, int lane)
{
    const int r = item / segs, sg = item - r * segs;
    if constexpr (sizeof(T) == 2) {
        x.j = 1 + r;
        x.i = 2 * (32 * sg + lane);
        x.w0 = x.i >= 1 && x.i <= a.nx - 2 && !in_tile(ib, pr, x.i, x.j);
        x.w1 = x.i + 1 <= a.nx - 2 && !in_tile(ib, pr, x.i + 1, x.j);
    } else {
        x.j = sizeof(T) == 4 ? 1 + 2 * r : 1 + r;
        x.i = 32 * sg + lane;
        const bool in = x.i >= 1 && x.i <= a.nx - 2;
        x.w0 = in && !in_tile(ib, pr, x.i, x.j);
        x.w1 = sizeof(T) == 4 && in && x.j + 1 <= a.ny - 2 && !in_tile(ib, pr, x.i, x.j + 1);
    }
}

// the lane's populations from the stage
template <typename T> __device__ __forceinline__ void item_read(LatticeItem<T> &x, const unsigned char *stage, int lane)
{
    using I = Items<T>;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const unsigned char *seg = stage + 16 * I::at(k);
        if constexpr (sizeof(T) == 2) {
            const uint32_t *w = reinterpret_cast<const uint32_t *>(seg) + lane;
            uint32_t v;
            if (lbm_ex(k) == 0) v = w[0];
            else if (lbm_ex(k) == 1) v = __byte_perm(w[I::AL / 2 - 1], w[I::AL / 2], 0x5432);   // columns i-1, i
            else v = __byte_perm(w[0], w[1], 0x5432);                                           // columns i+1, i+2
            x.g[k] = Pair2<T>::unpack(v);
        } else {
            const T *e = reinterpret_cast<const T *>(seg) + lane + (lbm_ex(k) == 1 ? I::AL - 1 : (lbm_ex(k) == -1 ? 1 : 0));
            if constexpr (sizeof(T) == 4) x.g[k] = make_float2(e[0], e[4 * I::ROW]);
            else x.g[k] = e[0];
        }
    }
}

template <typename T, typename C, bool CONS0>
__device__ __forceinline__ void item_update(const LatticeItem<T> &x, const KFArgs<C> &a, T *fout, C *fl)
{
    if (!x.w0 && !x.w1) return;
    if constexpr (sizeof(T) == 8) {
        C o[9], rho, u, v;
        collide_interior<C, CONS0>(a, x.g, false, C(0), C(0), o, rho, u, v);
        put_node<T, C>(a, fout, fl, x.i, x.j, o, rho, u, v);
    } else {
        constexpr bool XPAIR = sizeof(T) == 2;
        const int pitch = a.pitch, plane = (int)a.plane, d = XPAIR ? 1 : pitch;   // to the second node
        float2 o[9], rho, u, v;
        if (fl) collide_pair<CONS0, true>(a, x.g, o, rho, u, v);
        else collide_pair<CONS0, false>(a, x.g, o, rho, u, v);
        T *q = fout + x.j * pitch + x.i;
        if (XPAIR && x.w0 && x.w1) {
            if constexpr (XPAIR) {
#pragma unroll
                for (int k = 0; k < 9; ++k) *reinterpret_cast<uint32_t *>(q + k * plane) = Pair2<T>::pack(o[k]);
            }
        } else {
            if (x.w0) {
#pragma unroll
                for (int k = 0; k < 9; ++k) q[k * plane] = Store<T>::pack(o[k].x);
            }
            if (x.w1) {
#pragma unroll
                for (int k = 0; k < 9; ++k) q[k * plane + d] = Store<T>::pack(o[k].y);
            }
        }
        if (fl) {
            const long long nn = (long long)a.nx * a.ny, n0 = (long long)x.j * a.nx + x.i;
            if (x.w0) put_fields(fl, nn, n0, rho.x, u.x, v.x);
            if (x.w1) put_fields(fl, nn, n0 + (XPAIR ? 1 : a.nx), rho.y, u.y, v.y);
        }
    }
}

// node e of the lattice's edge, 0 <= e < 2 nx + 2 (ny - 2)
template <typename T, typename C>
__device__ __forceinline__ void edge_node(const KFArgs<C> &a, const T *fin, T *fout, C *fl, int e)
{
    int i, j;
    if (e < 2 * a.nx) {
        i = e >> 1;
        j = (e & 1) ? a.ny - 1 : 0;
    } else {
        j = 1 + ((e - 2 * a.nx) >> 1);
        i = (e & 1) ? a.nx - 1 : 0;
    }
    C o[9], rho, u, v;
    edge_update<T, C, LdCg>(a, fin, i, j, o, rho, u, v);
    put_node<T, C>(a, fout, fl, i, j, o, rho, u, v);
}

// warps of the solver: one per even block of the first level (and a thread
// per marker); more would only lengthen its barriers
__device__ __forceinline__ int solver_warps(int nb) { return max(4, (nb + 1) / 2); }

// The solver CTA's steps. Dynamic shared memory: the step's factor blocks
// (block o at index o), the right-hand sides in the solve order, an mbarrier.
template <typename C>
__device__ __forceinline__ void solver_cta(const LoopArgs<C> &L, double *smem)
{
    const int n = L.ib.nseg, nb = (n + BS - 1) / BS, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int NW = min(solver_warps(nb), (int)blockDim.x / 32), NT = 32 * NW;
    if (warp >= NW) return;   // barriers below count the threads that have not exited
    double *stage = smem, *X = smem + nb * BS * GW;
    uint64_t *bar = reinterpret_cast<uint64_t *>(X + 2 * nb * BS);
    // block o at index o; block 0 only its D_0^-1, whose rows (read in one
    // step, like columns of the others) are kept apart by banks
    constexpr uint32_t kBlock = sizeof(double) * BS * GW, kRow = sizeof(double) * BS;
    constexpr int ROOT_LD = BS + 2;
    if (tid == 0) {
        mbar_init(bar, 1);
        mbar_init_fence();
    }
    __syncthreads();
    uint32_t parity = 0;
    // warp 0, once the CTA is done with the previous step's factor blocks:
    // the copies of step s
    auto issue = [&](int s) {
        const IBArgs a = step_args(L.ib, L.step0 + s);
        if (warp != 0 || a.fmode[0]) return;
        if (lane == 0) mbar_expect_tx(bar, kBlock * (uint32_t)(nb - 1) + kRow * BS);
        __syncwarp();
        fence_proxy_async();
        if (lane < BS) bulk_g2s(stage + lane * ROOT_LD, a.gf + lane * GW, kRow, bar);   // D_0^-1
        for (int m = 1 + lane; m < nb; m += 32) bulk_g2s(stage + m * BS * GW, a.gf + (long long)m * BS * GW, kBlock, bar);
    };
    issue(0);
    for (int s = 0; s < L.nsteps; ++s) {
        const IBArgs a = step_args(L.ib, L.step0 + s);
        const bool dense = a.fmode[0] != 0;
        if (tid == 0) {
            const unsigned fs = *a.fstatus;
            if (fs) { atomicOr(a.status, fs); *a.fstatus = 0u; }
            a.solve_res[1] = (double)a.fmode[1];
        }
        bool ok = true;
        if (!dense) {   // the factor blocks
            int spins = 0;
            while (!mbar_try_wait(bar, parity))
                if (++spins > SPINS) {
                    ok = false;
                    break;
                }
            if (!ok) {   // report, then wait (bounded) for the copies still in flight
                give_up(L.sync, a.status);
                for (spins = 0; !mbar_try_wait(bar, parity) && spins < SPINS; ++spins) {
                }
            }
            parity ^= 1u;
        }
        // the right-hand sides in the solve order, each as soon as it is
        // there (16-byte pairs; the dense solve keeps the two apart)
        const int np = dense ? n : nb * BS;
        for (int q = tid; q < np && ok; q += NT) {
            double x = 0.0, y = 0.0;
            if (q < n) ok = wait_pair(a.rhs + 2 * q, L.sync, a.status, x, y);
            X[dense ? q : 2 * q] = x;
            X[dense ? n + q : 2 * q + 1] = y;
        }
        if (__syncthreads_or(!ok)) return;
        if (dense) {
            dense_tri(a, X, NT);
            __syncthreads();
        } else {
            // the levels with more than one even block
            int st = 1;
            for (; 2 * st < nb; st <<= 1) {
                for (int e = 2 * st * warp; e < nb; e += 2 * st * NW)
                    bcr_forward(stage + (e + st) * BS * GW, stage + (e - st) * BS * GW, X, e, st, e + st < nb, e > 0, lane);
                __syncthreads();
            }
            // two blocks are left, 0 and st (or one): warp 0's alone
            if (warp == 0) {
                if (st < nb) bcr_forward(stage + st * BS * GW, stage, X, 0, st, true, false, lane);
                __syncwarp();
                bcr_root(stage, ROOT_LD, X, lane);
                __syncwarp();
                if (st < nb) bcr_backward(stage + st * BS * GW, X, st, st, false, lane);
            }
            __syncthreads();
            for (st >>= 1; st > 0; st >>= 1) {
                for (int o = st * (2 * warp + 1); o < nb; o += 2 * st * NW)
                    bcr_backward(stage + o * BS * GW, X, o, st, o + st < nb, lane);
                __syncthreads();
            }
        }
        for (int q = tid; q < n; q += NT) {
            put_value(a.y + 2 * q, X[dense ? q : 2 * q]);
            put_value(a.y + 2 * q + 1, X[dense ? n + q : 2 * q + 1]);
        }
        __syncthreads();
        if (s + 1 < L.nsteps) issue(s + 1);
    }
}

// One case (MULTI false: its arguments are L0, its CTAs the grid), or a batch
// of cases (CTA b: entry b of `map`, {case, its CTA, its CTAs}), which share
// the launch and nothing else.
template <typename T, typename C, bool CONS0, bool MULTI>
__global__ void __launch_bounds__(NT, 1) step_loop(const __grid_constant__ LoopArgs<C> L0, const LoopArgs<C> *cases,
                                                   const int4 *map)
{
    constexpr int NW = NT / 32, NG = NT / TILE_THREADS;
    extern __shared__ __align__(128) double smem[];
    // a batch's arguments are read in shared memory: in global memory every
    // store might alias them
    __shared__ __align__(16) uint32_t lw[MULTI ? sizeof(LoopArgs<C>) / 4 : 1];
    int me = blockIdx.x, all = gridDim.x;
    if (MULTI) {
        const int4 m = map[blockIdx.x];
        me = m.y;
        all = m.z;
        const uint32_t *src = reinterpret_cast<const uint32_t *>(cases + m.x);
        for (int w = threadIdx.x; w < (int)(sizeof(LoopArgs<C>) / 4); w += NT) lw[w] = src[w];
        __syncthreads();
    }
    const LoopArgs<C> &L = MULTI ? *reinterpret_cast<const LoopArgs<C> *>(lw) : L0;
    if (me == 0) {
        solver_cta<C>(L, smem);
        return;
    }
    __shared__ int good[NG], taken[2];   // taken: the interior items of the step (by parity)
    const int cta = me - 1, G = all - 1;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int grp = tid / TILE_THREADS, gt = tid % TILE_THREADS;
    if (gt == 0) good[grp] = 1;
    group_sync(grp);
    const KFArgs<C> &kf = L.kf;
    TileSmem &S = reinterpret_cast<GroupSmem *>(smem)[grp].tile;
    TileWeights &W = reinterpret_cast<GroupSmem *>(smem)[grp].weights;
    // the warp's stages of the lattice update, after the groups' tiles
    using I = Items<T>;
    static_assert(NG * sizeof(GroupSmem) + NW * I::STAGES * I::BYTES <= LOOP_SMEM, "shared memory");
    unsigned char *stage = reinterpret_cast<unsigned char *>(smem) + NG * sizeof(GroupSmem) + warp * I::STAGES * I::BYTES;
    __shared__ int tab[I::ROW];
    item_table<T>(tab, (int)kf.plane, kf.pitch);
    if (tid < 2) taken[tid] = 0;
    __syncthreads();
    const int n = L.ib.nseg, nx = kf.nx, ny = kf.ny;
    constexpr bool XPAIR = sizeof(T) == 2, YPAIR = sizeof(T) == 4;
    const int segs = XPAIR ? (nx + 63) / 64 : (nx + 31) / 32;
    const int items = segs * (YPAIR ? (ny - 1) / 2 : ny - 2);
    const int nedge = 2 * nx + 2 * (ny - 2), nthr = G * NT;
    // The CTA's two groups of TILE_THREADS threads work apart from each other.
    // Correction tiles go to the CTAs from the last one on, in turn to the one
    // or the other group from step to step: the group that has no tiles in a
    // step prepares those of the next one as soon as its part of the step is
    // done. Markers go to the CTAs from the first one on that have no tile
    // (but to half of the CTAs at least); the first marker's weights are
    // loaded a step ahead.
    auto tiles_of = [&](const IBArgs &a) -> int {
        const int c = *a.nsup;
        if (c >= 0 && c <= patch_tiles(a)) return c;
        if (tid == 0) atomicOr(a.status, LBM_ST_INDEX_TILE);
        return 0;
    };
    auto marker_ctas = [&](int ntile) { return max(G - ntile, (G + 1) / 2); };
    IBArgs a = step_args(L.ib, L.step0);
    int ntile = tiles_of(a), mctas = marker_ctas(ntile);
    int k0 = cta < mctas ? warp * mctas + cta : n;
    InterpLane il;
    if (k0 < n) il = interp_lane(a, k0, lane);
    // the tile in hand: node, markers, populations, correction
    int tile = -1, gi = 0, gj = 0, listed = 0, mark = -1, wing = 0, cnt = 0;
    bool active = false;
    C g[9];
    NodeMoments<C> q;
    double du = 0.0, dv = 0.0;
    auto forces = [&](const IBArgs &a) {
        const bool sup = active && wing < (1 << 20);
        double fx = 0.0, fy = 0.0, mz = 0.0;
        if (sup) node_force(a, motion_row(a, a.cur_step, nullptr), g, gi, gj, wing, du, dv, fx, fy, mz);
        tile_force_warp(a, S, sup, wing, fx, fy, mz, gt >> 5, lane);
        group_sync(grp);
        tile_force_store(a, S, tile, gt);
    };
    // the markers of correction tile c, and the weights with which they act on
    // the thread's node
    auto prepare = [&](int c) {
        const int nt = patch_tiles(a);
        const PatchInfo pr = *a.pinfo;
        tile = a.ctile[c];
        if (tile < 0 || tile >= nt) {
            if (gt == 0) atomicOr(a.status, LBM_ST_INDEX_TILE);
            tile = -1;   // the same for the whole group
            return;
        }
        const int ti0 = (tile % a.tiles_x) * TILE, tj0 = (tile / a.tiles_x) * TILE;
        const int li = ti0 + (gt & 15), lj = tj0 + (gt >> 4);
        gi = pr.i0 + li;
        gj = pr.j0 + lj;
        active = li < pr.w && lj < pr.h;
        if (active && (gi < 1 || gi > nx - 2 || gj < 1 || gj > ny - 2)) {
            atomicOr(a.status, LBM_ST_INDEX_TILE);
            active = false;
        }
        const int *tl = a.tiles + (long long)tile * (TILE_CAP + 1);
        listed = tl[0];
        mark = -1;
        if (listed <= TILE_CAP && gt < listed) {
            mark = tl[1 + gt];
            mark = tile_stage(a, S, gt, mark) ? tile_position(a, mark) : -1;
        }
        group_sync(grp);
        wing = 1 << 20;
        cnt = listed <= TILE_CAP ? tile_cover(S, W, listed, active, gi, gj, gt, wing) : 0;
    };
    const int c0 = G - 1 - cta;   // the CTA's first tile
    if (grp == 0 && c0 < ntile) prepare(c0);
    for (int s = 0; s < L.nsteps; ++s) {
        const T *fin = (const T *)L.f[s & 1];
        T *fout = (T *)L.f[(s & 1) ^ 1];
        C *fl = L.fields[s];
        const bool duty = (s & 1) == grp;
        if (tid == 0) taken[(s & 1) ^ 1] = 0;   // nobody takes of it before the next step
        for (int k = k0; k < n; k += NW * mctas) {
            if (k > k0) il = interp_lane(a, k, lane);
            double ru, rv;
            interp_sum<T, LdCg>(a, fin, il, ru, rv);
            if (lane == 0 && il.pos >= 0) {
                put_value(a.rhs + 2 * il.pos, ru);
                put_value(a.rhs + 2 * il.pos + 1, rv);
            }
        }
        // while the solver works: the nodes outside the correction tiles, edge
        // nodes and interior, each dealt out from the group without tiles on
        const PatchInfo pr = *a.pinfo;
        const int et = duty ? TILE_THREADS + gt : gt;   // thread of the CTA, the free group first
        for (int e = (TILE_THREADS - 1 - et + (duty ? NT : 0)) * G + cta; e < nedge; e += nthr) edge_node<T, C>(kf, fin, fout, fl, e);
        // The CTA's interior items (`mine`): a CTA with a tile in this step has
        // LEAN less than the others, none on a small lattice. The first `dealt`
        // of them are dealt out to the warps; the last (TAIL a warp) go to the
        // warps as they come, since a group that was still preparing a tile
        // when the step began is behind.
        const int nn = G - min(ntile, G);   // CTAs without a tile, the first ones
        const int each = nn > 0 ? max(0, (items - LEAN * nn) / G) : (items + G - 1) / G;
        const int mine = cta < nn ? each + (items - each * G - cta + nn - 1) / nn : each;
        const int dealt = mine > NW ? max(0, mine / NW - TAIL) * NW : mine;
        int turn = et >> 5;   // the free group first
        auto take = [&]() -> int {
            int q = turn;
            if (q < dealt) {
                turn += NW;
            } else {
                if (mine > NW) {
                    if (lane == 0) q = atomicAdd(&taken[s & 1], 1);
                    q = dealt + __shfl_sync(0xffffffffu, q, 0);
                }
                if (q >= mine) return items;
            }
            return q < each ? q * G + cta : each * G + (q - each) * nn + cta;
        };
        int it[I::STAGES];
#pragma unroll
        for (int t = 0; t < I::STAGES - 1; ++t) {
            it[t] = take();
            if (it[t] < items) item_issue<T, C>(kf, fin, tab, stage + t * I::BYTES, it[t], segs, lane);
            copies_commit();
        }
        for (int q = 0; it[0] < items;) {
            const int qn = q == 0 ? I::STAGES - 1 : q - 1;
            it[I::STAGES - 1] = take();
            if (it[I::STAGES - 1] < items) item_issue<T, C>(kf, fin, tab, stage + qn * I::BYTES, it[I::STAGES - 1], segs, lane);
            copies_commit();
            LatticeItem<T> x;
            item_nodes<T, C>(x, kf, a, pr, it[0], segs, lane);
            copies_wait<I::STAGES - 1>();
            __syncwarp();
            item_read<T>(x, stage + q * I::BYTES, lane);
            __syncwarp();
            item_update<T, C, CONS0>(x, kf, fout, fl);
            q = q + 1 == I::STAGES ? 0 : q + 1;
#pragma unroll
            for (int t = 0; t < I::STAGES - 1; ++t) it[t] = it[t + 1];
        }
        // the update of the prepared tile; what its forces need is kept
        auto update = [&]() {
            du = dv = 0.0;
            if (active) {
                pull<T, C, LdCg>(fin, kf.plane, kf.pitch, gi, gj, g);
                q = node_moments_of(g);
            }
            if (listed <= TILE_CAP) {
                if (mark >= 0) {
                    double x = 0.0, y = 0.0;
                    if (!wait_pair(a.y + 2 * mark, L.sync, a.status, x, y)) good[grp] = 0;
                    S.y[gt][0] = x;
                    S.y[gt][1] = y;
                } else if (gt < listed) {
                    S.y[gt][0] = S.y[gt][1] = 0.0;
                }
                group_sync(grp);
                if (active) tile_sum(S, W, cnt, listed, gi, gj, gt, du, dv);
            } else {
                // more markers than a list holds: scan all of them, in order
                const int ti0 = (tile % a.tiles_x) * TILE, tj0 = (tile / a.tiles_x) * TILE;
                const int ta = pr.i0 + ti0, tb = ta + TILE - 1, sa = pr.j0 + tj0, sb = sa + TILE - 1;
                const int gw = gt >> 5;
                for (int m0 = 0; m0 < n; m0 += TILE_THREADS) {
                    const int k = m0 + gt;
                    bool hit = false;
                    if (k < n) {
                        if (marker_ok(a, a.mk[k])) {
                            const int4 b = mbox(a.mk[k]);
                            hit = b.x <= tb && b.y >= ta && b.z <= sb && b.w >= sa && b.y >= b.x;
                        } else {
                            atomicOr(a.status, LBM_ST_INDEX_TILE);
                        }
                    }
                    const unsigned bal = __ballot_sync(0xffffffffu, hit);
                    if (lane == 0) S.wsum[gw] = __popc(bal);
                    group_sync(grp);
                    int before = 0, all = 0;
                    for (int w = 0; w < 8; ++w) {
                        const int t = S.wsum[w];
                        before += w < gw ? t : 0;
                        all += t;
                    }
                    if (hit) {
                        const int at = before + __popc(bal & ((1u << lane) - 1u));
                        const int pos = tile_stage(a, S, at, k) ? tile_position(a, k) : -1;
                        double x = 0.0, y = 0.0;
                        if (pos >= 0 && !wait_pair(a.y + 2 * pos, L.sync, a.status, x, y)) good[grp] = 0;
                        S.y[at][0] = x;
                        S.y[at][1] = y;
                    }
                    group_sync(grp);
                    if (active) tile_gather(S, 0, all, gi, gj, du, dv, wing);
                    group_sync(grp);
                }
            }
            if (active) {
                C o[9], rho, u, v;
                collide_moments<C>(kf, g, q, true, (C)du, (C)dv, o, rho, u, v);
                put_node<T, C>(kf, fout, fl, gi, gj, o, rho, u, v);
            }
        };
        if (duty)
            for (int c = c0; c < ntile; c += G) {
                if (c > c0) {
                    if (tile >= 0) forces(a);
                    group_sync(grp);
                    prepare(c);
                }
                if (tile >= 0) update();
            }
        // the group's part of the step is handed on
        group_sync(grp);
        if (gt == 0) red_release(L.sync + SYNC_STEP, 1u);
        if (!good[grp]) return;
        if (duty && c0 < ntile && tile >= 0) forces(a);
        if (s + 1 == L.nsteps) return;
        // what the next step needs ahead of its start
        a = step_args(L.ib, L.step0 + s + 1);
        ntile = tiles_of(a);
        mctas = marker_ctas(ntile);
        k0 = cta < mctas ? warp * mctas + cta : n;
        if (k0 < n) il = interp_lane(a, k0, lane);
        if (!duty && c0 < ntile) prepare(c0);
        if (gt == 0) good[grp] = wait_step(L.sync, L.base + (unsigned)(NG * G) * (unsigned)(s + 1), a.status);
        group_sync(grp);
        if (!good[grp]) return;
    }
}

size_t loop_smem(const lbm_handle *h)
{
    const size_t nb = (size_t)(h->nseg + BS - 1) / BS;
    const size_t solve = sizeof(double) * (nb * BS * GW + 2 * nb * BS) + 16;
    const size_t stages = h->elem == 2 ? Items<__half>::STAGES * Items<__half>::BYTES
                          : h->elem == 4 ? Items<float>::STAGES * Items<float>::BYTES : Items<double>::STAGES * Items<double>::BYTES;
    return std::max(solve, NT / TILE_THREADS * sizeof(GroupSmem) + NT / 32 * stages);
}

// nodes (or pairs) of a lattice
int loop_units(const lbm_handle *h) { return h->nx * h->ny / (h->elem == 8 ? 1 : 2); }

// CTAs beside the solver that a case's lattice can use: one group's threads
// for every 256 nodes (or pairs), so that the group without tiles does the
// lattice alone where the SMs suffice; fewer than 24 CTAs leave tiles to
// share one (96x64: 10.0 us a step on 6 CTAs, 9.1 on 24 and on 132)
int loop_want(const lbm_handle *h)
{
    return std::max((loop_units(h) + TILE_THREADS - 1) / TILE_THREADS, 24);
}

template <typename C>
LoopArgs<C> loop_args(lbm_handle *h, int nsteps, void *const *fields, int ring_slot, bool check_last)
{
    LoopArgs<C> L;
    ib_args_write(h, nullptr, 0, &L.ib);
    L.ib.ring_row = ring_slot;
    L.ib.check_res = check_last;
    L.kf = make_kf_args<C>(h, nullptr, nullptr, nullptr, KF_OUTER);
    L.f[0] = h->fbuf[h->cur];
    L.f[1] = h->fbuf[h->cur ^ 1];
    for (int s = 0; s < LOOP_STEPS; ++s) L.fields[s] = fields && s < nsteps ? (C *)fields[s] : nullptr;
    L.step0 = h->n;
    L.nsteps = nsteps;
    L.sync = h->d_sync;
    // every launch adds the same number to the step counter, whatever it
    // waited for; after one that gave up the counters start over (loop_reset)
    L.base = h->sync_base;
    return L;
}

// the launch of `ctas` CTAs for a case is accounted for
void loop_done(lbm_handle *h, int ctas, int nsteps)
{
    h->sync_base += (unsigned)(NT / TILE_THREADS * (ctas - 1) * nsteps);
    h->count(4ll * nsteps, 1);   // interpolation, solve, lattice, correction tiles of each step
}

template <typename T, typename C, bool CONS0>
int launch_loop_t(lbm_handle *h, int nsteps, void *const *fields, cudaStream_t st)
{
    LoopArgs<C> L = loop_args<C>(h, nsteps, fields, 0, false);
    const size_t smem = loop_smem(h);
    auto kernel = step_loop<T, C, CONS0, false>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LOOP_SMEM) != cudaSuccess) return -1;
    const int ctas = std::min(1 + loop_want(h), h->loop_ctas);
    const LoopArgs<C> *cases = nullptr;
    const int4 *map = nullptr;
    void *args[] = {&L, &cases, &map};
    if (cudaLaunchCooperativeKernel((const void *)kernel, dim3(ctas), dim3(NT), args, smem, st) != cudaSuccess) return -1;
    loop_done(h, ctas, nsteps);
    return 0;
}

template <typename T, typename C, bool CONS0>
int launch_loop_multi_t(int ctas, size_t smem, const void *dcases, const int4 *dmap, cudaStream_t st)
{
    auto kernel = step_loop<T, C, CONS0, true>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LOOP_SMEM) != cudaSuccess) return -1;
    LoopArgs<C> none{};
    const LoopArgs<C> *cases = (const LoopArgs<C> *)dcases;
    void *args[] = {&none, &cases, &dmap};
    return cudaLaunchCooperativeKernel((const void *)kernel, dim3(ctas), dim3(NT), args, smem, st) == cudaSuccess ? 0 : -1;
}

// bytes by which the lattices of a loop are measured: 2-byte storage counts as
// 4-byte (its update is bound by the nodes)
long long loop_bytes(const lbm_handle *h) { return 18ll * std::max<long long>(4, (long long)h->elem) * h->plane; }

}  // namespace

int loop_sync_words() { return SYNC_WORDS; }

cudaError_t loop_reset(lbm_handle *h)
{
    h->sync_base = 0;
    return cudaMemsetAsync(h->d_sync, 0, SYNC_WORDS * sizeof(unsigned), h->stream);
}

// Whether a handle's steps run as step_loop launches.
bool loop_fits(const lbm_handle *h)
{
    if (h->loop_ctas < 2 || h->nseg <= 0 || h->nslots / 2 > LOOP_STEPS || loop_smem(h) > LOOP_SMEM) return false;
    // Beyond these two steps in one pass (kf_pair) are faster, in FP64 earlier
    // (the loop's lattice update is then bound by the FP64 units and the L2).
    // us a step, here and there: FP32 2048x1024 (151 MB) 32 and 39, 2400x1200
    // (207 MB) 41 and 42; FP16 2048x1024 26 and 37; FP64 1200x600 (104 MB) 27
    // and 34, 1400x700 (141 MB) 37.5 and 34.6, 1600x800 (184 MB) 47 and 39.
    return loop_bytes(h) <= (h->elem == 8 ? 125000000ll : 220000000ll);
}

// `nsteps` steps from step h->n on (within one slot half), step s with its
// fields written to fields[s] unless null
int launch_loop(lbm_handle *h, int nsteps, void *const *fields, cudaStream_t st)
{
    const bool c0 = h->s[0] == 0.0 && h->s[3] == 0.0 && h->s[5] == 0.0;
    switch (h->prec) {
    case LBM_PREC_FP32:
        return c0 ? launch_loop_t<float, float, true>(h, nsteps, fields, st) : launch_loop_t<float, float, false>(h, nsteps, fields, st);
    case LBM_PREC_FP64:
        return c0 ? launch_loop_t<double, double, true>(h, nsteps, fields, st) : launch_loop_t<double, double, false>(h, nsteps, fields, st);
    case LBM_PREC_FP16:
        return c0 ? launch_loop_t<__half, float, true>(h, nsteps, fields, st) : launch_loop_t<__half, float, false>(h, nsteps, fields, st);
    case LBM_PREC_BF16:
        return c0 ? launch_loop_t<__nv_bfloat16, float, true>(h, nsteps, fields, st) : launch_loop_t<__nv_bfloat16, float, false>(h, nsteps, fields, st);
    }
    return -1;
}

// ---- a batch of cases --------------------------------------------------------

size_t loop_args_size(int prec) { return prec == LBM_PREC_FP64 ? sizeof(LoopArgs<double>) : sizeof(LoopArgs<float>); }

void loop_args_write(lbm_handle *h, int nsteps, void *const *fields, int ring_slot, bool check_last, void *dst)
{
    if (h->prec == LBM_PREC_FP64)
        *(LoopArgs<double> *)dst = loop_args<double>(h, nsteps, fields, ring_slot, check_last);
    else
        *(LoopArgs<float> *)dst = loop_args<float>(h, nsteps, fields, ring_slot, check_last);
}

// The CTAs of each case when `hs` run as one step_loop launch (empty: they
// do not): one solver and at least one more, the rest by lattice size. Launches
// per stage cost a batch some 20 us a step and 0.5 us a case before any
// lattice, a shared launch nothing, but it has 132 CTAs for all, which take
// each their part of a lattice at 3.4 ns a node, however idle the others are:
// the more cases, the fewer nodes (pairs, in FP32) a CTA may be left with.
// us a step, launches per stage and here: 256x128, 32 cases (5461 a CTA) 54 and
// 52, 36 (8192) 59 and 67, 48 (16384) 74 and 122; 384x192, 20 cases (7373) 59
// and 55, 28 (12288) 74 and 81; 160x96, 40 (3840) 56 and 56, 48 (7680) 63 and
// 89; 96x64, 48 to 66 (3072) 55 to 68 either way; FP64 160x96, 32 (5120) 57 and
// 56, 48 (15360) 77 and 139. By bytes: 512x256, 12 cases (113 MB) 54 and 45, 16
// (151 MB) 66 and 62, 20 (189 MB) 76 and 81; 800x400, 4 (92 MB) 43 and 31, 12
// (276 MB) 87 and 91.
std::vector<int> loop_shares(lbm_handle *const *hs, int n)
{
    std::vector<int> share;
    if (n < 1) return share;
    const int total = hs[0]->loop_ctas;
    long long bytes = 0;
    double units = 0.0;
    for (int c = 0; c < n; ++c) {
        if (!loop_fits(hs[c])) return share;
        bytes += loop_bytes(hs[c]);
        units += (double)loop_want(hs[c]);
    }
    if (2 * n > total || bytes > 150000000ll) return share;
    share.assign(n, 0);
    int used = 0, most = 0;   // most: nodes or pairs of a CTA
    for (int c = 0; c < n; ++c) {
        const int want = loop_want(hs[c]);
        const int work = std::max(1, std::min(want, (int)((total - 2 * n) * (want / units)) + 1));
        share[c] = 1 + work;
        used += share[c];
        most = std::max(most, loop_units(hs[c]) / work);
    }
    return used <= total && most <= std::max(4000, 16000 - 310 * n) ? share : std::vector<int>();
}

int launch_loop_multi(lbm_handle *const *hs, int n, const std::vector<int> &share, int nsteps, bool cons0,
                      const void *dcases, const int4 *dmap, cudaStream_t st)
{
    size_t smem = 0;
    int ctas = 0;
    for (int c = 0; c < n; ++c) {
        smem = std::max(smem, loop_smem(hs[c]));
        ctas += share[c];
    }
    int rc = -1;
    switch (hs[0]->prec) {
    case LBM_PREC_FP32:
        rc = cons0 ? launch_loop_multi_t<float, float, true>(ctas, smem, dcases, dmap, st) : launch_loop_multi_t<float, float, false>(ctas, smem, dcases, dmap, st);
        break;
    case LBM_PREC_FP64:
        rc = cons0 ? launch_loop_multi_t<double, double, true>(ctas, smem, dcases, dmap, st) : launch_loop_multi_t<double, double, false>(ctas, smem, dcases, dmap, st);
        break;
    case LBM_PREC_FP16:
        rc = cons0 ? launch_loop_multi_t<__half, float, true>(ctas, smem, dcases, dmap, st) : launch_loop_multi_t<__half, float, false>(ctas, smem, dcases, dmap, st);
        break;
    case LBM_PREC_BF16:
        rc = cons0 ? launch_loop_multi_t<__nv_bfloat16, float, true>(ctas, smem, dcases, dmap, st) : launch_loop_multi_t<__nv_bfloat16, float, false>(ctas, smem, dcases, dmap, st);
        break;
    }
    return rc;
}

void loop_account(lbm_handle *h, int ctas, int nsteps) { loop_done(h, ctas, nsteps); }
