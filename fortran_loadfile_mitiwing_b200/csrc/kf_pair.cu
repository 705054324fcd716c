// kf_pair.cu -- two time steps of a large lattice in one pass over memory.
//
// A step reads and writes every population once, and on a large lattice that
// traffic is its time. Away from the bodies and the edge two steps need
// nothing but the populations before them, so one CTA takes a node's
// neighbourhood through both: it stages the rows of its strip as the
// single-step kernel does, keeps the first step's results on chip (its own
// column's in registers, the neighbour columns' by shuffles), and writes only
// the second step's. The traffic per step is halved; the arithmetic grows by
// the two rows around a CTA's nodes and the two columns around a warp's that
// are computed for the first step only. 4096x2048, us a step, single-step
// kernel alone -> here: FP32 104 -> 54 (85 % of the copy bandwidth), FP16
// 60 -> 45, FP64 195 -> 104; the 2-byte form is bound by instruction issue.
//
// The nodes near a body go step by step: the first step's correction tiles
// and the nodes next to them depend on the first step's solve, the second
// step's tiles on the second one's. kf_near takes them through the steps
// between the immersed-boundary stages, with a third population buffer for
// the state in between, in units of 16 x 16 cells of the lattice (ib_near
// lists the cells that hold such a node), and with them the edge.
#include <algorithm>
#include <type_traits>

#include "ib_device.cuh"

namespace {

using namespace lbm_node;
using lbm_ib::TILE;
using lbm_ib::TILE_CAP;

constexpr int PT = 256;      // threads of a CTA
constexpr int CELL = 16;     // nodes of a cell's side
constexpr int FRAME = 2;     // nodes at the lattice's edge that kf_pair leaves (their second step needs the edge's first)

// rows of a strip staged ahead (4096x2048, us a step with 3, 4, 5: FP32 73.4,
// 72.0, 72.2, FP16 62.0, 60.9, 60.2: beyond 3 no more than the runs differ)
template <typename T> __host__ __device__ constexpr int pair_stages() { return 4; }

template <typename C> struct PairArgs {
    const void *fin;
    void *fout;
    int nx, ny, pitch;
    long long plane;
    C s[9], sc[9];
    int rows;                     // rows a CTA writes (even)
    const unsigned char *near;    // per cell of the lattice: left to kf_near
    int cells_x;
    unsigned *status;
};

// Columns that a CTA writes: 30 (2-byte storage: 30 pairs) of each warp. A
// warp computes the first step of one more on either side and gets the
// neighbours' first-step values by shuffles, so that the warps need no barrier
// among them in the row loop. (With 254 columns a CTA, the neighbours' values
// through shared memory and a barrier per row pair, the barrier was 40 % of
// the stalls; 4096x2048, us a pair of steps alone, then -> now: FP32 123 ->
// 109, FP16 100 -> 89.)
constexpr int WOUT = 30;
template <typename T> __host__ __device__ constexpr int pair_out() { return (sizeof(T) == 2 ? 2 : 1) * WOUT * (PT / 32); }
// columns of the first step
template <typename T> __host__ __device__ constexpr int pair_cols() { return pair_out<T>() + (sizeof(T) == 2 ? 4 : 2); }
template <typename T> __host__ __device__ constexpr int pair_align() { return 16 / (int)sizeof(T); }
// elements of a staged row segment: the columns, one or two more at each side,
// from a 16-byte boundary on
template <typename T> __host__ __device__ constexpr int pair_seg()
{
    return (pair_cols<T>() + pair_align<T>() - 1) / pair_align<T>() * pair_align<T>() + 2 * pair_align<T>();
}
template <typename T> __host__ __device__ constexpr size_t pair_smem()
{
    return sizeof(T) * pair_stages<T>() * 9 * pair_seg<T>() + 2 * 8 * pair_stages<T>();
}

// one node (or pair of nodes) of the first or second step
template <bool CONS0> __device__ __forceinline__ void pair_step(const KFArgs<float> &a, const float2 g[9], float2 o[9])
{
    float2 r, u, v;
    collide_pair<CONS0, false>(a, g, o, r, u, v);
}

// the value of the warp's left, right neighbour column
template <typename V> __device__ __forceinline__ V from_left(V v) { return __shfl_up_sync(0xffffffffu, v, 1); }
template <typename V> __device__ __forceinline__ V from_right(V v) { return __shfl_down_sync(0xffffffffu, v, 1); }
template <> __device__ __forceinline__ float2 from_left(float2 v) { return make_float2(from_left(v.x), from_left(v.y)); }
template <> __device__ __forceinline__ float2 from_right(float2 v) { return make_float2(from_right(v.x), from_right(v.y)); }

// One CTA: strip bx and row chunk by of the lattice described by p.
template <typename T, typename C, bool CONS0>
__device__ __forceinline__ void pair_cta(const PairArgs<C> &p, int bx, int by, unsigned char *sm)
{
    constexpr int SEG = pair_seg<T>(), KS = pair_stages<T>(), NWARP = PT / 32, AL = pair_align<T>();
    constexpr bool XPAIR = sizeof(T) == 2, YPAIR = sizeof(T) == 4;
    T *buf = reinterpret_cast<T *>(sm);
    uint64_t *full = reinterpret_cast<uint64_t *>(sm + sizeof(T) * KS * 9 * SEG);
    uint64_t *empty = full + KS;
    const int tid = threadIdx.x, lane = tid & 31;
    const int col = (tid >> 5) * WOUT + lane;      // of the first step (2-byte storage: pair of columns)
    // output columns from x0 on, first-step columns from x0 - 1 (x0 - 2) on
    const int x0 = FRAME + bx * pair_out<T>();
    const int xf = XPAIR ? x0 - 2 : x0 - 1;
    const int i = xf + (XPAIR ? 2 * col : col);
    const int y0 = FRAME + by * p.rows;
    const int nout = min(p.rows, p.ny - 2 - y0);   // rows written: y0 .. y0 + nout - 1 <= ny - 3
    const int nrows = nout + 2;                    // first-step rows y0 - 1 ..
    const int seg0 = (xf - 1) / AL * AL;           // staged columns from seg0 on (xf >= 1, or 0 where xf - 1 rounds up to 0)
    const int sh = xf - seg0;
    const int ncol = min(xf + pair_cols<T>() + 1, p.nx) - seg0;
    const uint32_t bytes = (uint32_t)((ncol * (int)sizeof(T) + 15) / 16 * 16);
    const T *__restrict__ fin = (const T *)p.fin;
    KFArgs<C> a;   // the constants of the collision
#pragma unroll
    for (int k = 0; k < 9; ++k) { a.s[k] = p.s[k]; a.sc[k] = p.sc[k]; }
    if (tid == 0) {
        for (int q = 0; q < KS; ++q) {
            mbar_init(&full[q], 1);
            mbar_init(&empty[q], NWARP);
        }
        mbar_init_fence();
    }
    __syncthreads();
    auto issue = [&](int r) {
        const int q = r % KS, j = y0 - 1 + r;
        mbar_expect_tx(&full[q], 9u * bytes);
#pragma unroll
        for (int k = 0; k < 9; ++k)
            bulk_g2s(buf + (q * 9 + k) * SEG, fin + (long long)k * p.plane + (long long)(j - lbm_ey(k)) * p.pitch + seg0, bytes,
                     &full[q]);
    };
    auto wait = [&](uint64_t *bar, uint32_t parity) -> bool {
        int spins = 0;
        while (!mbar_try_wait(bar, parity))
            if (++spins > (1 << 22)) return false;
        return true;
    };
    bool ok = true;
    // warp 0's refill of row r's stage with row r + KS
    auto refill = [&](int r) {
        if (tid == 0 && r + KS < nrows && ok) {
            ok = wait(&empty[r % KS], (uint32_t)((r / KS) & 1));
            if (ok) {
                fence_proxy_async();
                issue(r + KS);
            }
        }
    };
    if (tid == 0)
        for (int r = 0; r < KS && r < nrows; ++r) issue(r);
    // does any near cell meet the CTA's nodes?
    bool some = false;
    {
        const int c0 = x0 >> 4, c1 = min(x0 + pair_out<T>() - 1, p.nx - 3) >> 4, r0 = y0 >> 4, r1 = (y0 + nout - 1) >> 4;
        const int w = c1 - c0 + 1, n = w * (r1 - r0 + 1);
        for (int t = tid; t < n; t += PT) some = some || p.near[(r0 + t / w) * p.cells_x + c0 + t % w];
        some = __syncthreads_or(some);
    }
    T *const fout = (T *)p.fout;
    const bool out0 = lane > 0 && lane <= WOUT && i <= p.nx - 3;
    auto kept = [&](int ii, int j) { return some && p.near[(j >> 4) * p.cells_x + (ii >> 4)] != 0; };
    if constexpr (YPAIR) {
        float2 p0, p2, n1, n3, n5, n6;   // the iteration before: own column's planes 0, 2; neighbours' 1, 3, 5, 6
        p0 = p2 = n1 = n3 = n5 = n6 = make_float2(0.f, 0.f);
        for (int r = 0; r < nrows; r += 2) {
            const int r1 = min(r + 1, nrows - 1), q0 = r % KS, q1 = r1 % KS;
            bool got = wait(&full[q0], (uint32_t)((r / KS) & 1));
            got = wait(&full[q1], (uint32_t)((r1 / KS) & 1)) && got;
            ok = ok && got;
            float2 g[9], o[9];
            const T *b0 = buf + q0 * 9 * SEG + sh + col, *b1 = buf + q1 * 9 * SEG + sh + col;
#pragma unroll
            for (int k = 0; k < 9; ++k) g[k] = make_float2(b0[k * SEG - lbm_ex(k)], b1[k * SEG - lbm_ex(k)]);
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&empty[q0]);
                if (r1 != r) mbar_arrive(&empty[q1]);
            }
            pair_step<CONS0>(a, g, o);
            refill(r);
            if (r1 != r) refill(r1);
            if (!__all_sync(0xffffffffu, ok)) break;
            const float2 c1 = from_left(o[1]), c3 = from_right(o[3]), c5 = from_left(o[5]), c6 = from_right(o[6]);
            const float2 c7 = from_right(o[7]), c8 = from_left(o[8]);
            if (r > 0) {
                // rows (y0 - 1 + r) - 1 and y0 - 1 + r
                const int j = y0 - 2 + r;
                g[0] = make_float2(p0.y, o[0].x);
                g[1] = make_float2(n1.y, c1.x);
                g[2] = p2;
                g[3] = make_float2(n3.y, c3.x);
                g[4] = o[4];
                g[5] = n5;
                g[6] = n6;
                g[7] = c7;
                g[8] = c8;
                float2 w[9];
                pair_step<CONS0>(a, g, w);
                const bool s0 = out0 && !kept(i, j), s1 = out0 && j + 1 < y0 + nout && !kept(i, j + 1);
                const unsigned at = (unsigned)(j * p.pitch + i);
                if (s0) {
#pragma unroll
                    for (int k = 0; k < 9; ++k) (fout + (long long)k * p.plane)[at] = w[k].x;
                }
                if (s1) {
#pragma unroll
                    for (int k = 0; k < 9; ++k) (fout + (long long)k * p.plane + p.pitch)[at] = w[k].y;
                }
            }
            p0 = o[0]; p2 = o[2]; n1 = c1; n3 = c3; n5 = c5; n6 = c6;
        }
    } else if constexpr (XPAIR) {
        // words of two columns; q1, q3: pulled planes 1 and 3 of the row before,
        // q5, q6, p2: of the two rows before
        uint32_t p0 = 0, p2 = 0, p2b = 0, q1 = 0, q3 = 0, q5 = 0, q5b = 0, q6 = 0, q6b = 0;
        for (int r = 0; r < nrows; ++r) {
            const int q = r % KS;
            ok = wait(&full[q], (uint32_t)((r / KS) & 1)) && ok;
            float2 g[9], o[9];
            const uint32_t *b = reinterpret_cast<const uint32_t *>(buf + q * 9 * SEG + sh) + col;
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                const uint32_t *wk = b + k * (SEG / 2);
                uint32_t w;
                if (lbm_ex(k) == 0) w = wk[0];
                else if (lbm_ex(k) == 1) w = __byte_perm(wk[-1], wk[0], 0x5432);
                else w = __byte_perm(wk[0], wk[1], 0x5432);
                g[k] = Pair2<T>::unpack(w);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[q]);
            pair_step<CONS0>(a, g, o);
            uint32_t w[9];
#pragma unroll
            for (int k = 0; k < 9; ++k) w[k] = Pair2<T>::pack(o[k]);
            refill(r);
            if (!__all_sync(0xffffffffu, ok)) break;
            const uint32_t c1 = __byte_perm(from_left(w[1]), w[1], 0x5432), c3 = __byte_perm(w[3], from_right(w[3]), 0x5432);
            const uint32_t c5 = __byte_perm(from_left(w[5]), w[5], 0x5432), c6 = __byte_perm(w[6], from_right(w[6]), 0x5432);
            const uint32_t c7 = __byte_perm(w[7], from_right(w[7]), 0x5432), c8 = __byte_perm(from_left(w[8]), w[8], 0x5432);
            if (r > 1) {
                const int j = y0 - 2 + r;
                g[0] = Pair2<T>::unpack(p0);
                g[1] = Pair2<T>::unpack(q1);
                g[2] = Pair2<T>::unpack(p2b);
                g[3] = Pair2<T>::unpack(q3);
                g[4] = Pair2<T>::unpack(w[4]);
                g[5] = Pair2<T>::unpack(q5b);
                g[6] = Pair2<T>::unpack(q6b);
                g[7] = Pair2<T>::unpack(c7);
                g[8] = Pair2<T>::unpack(c8);
                pair_step<CONS0>(a, g, o);
                const bool s0 = out0 && !kept(i, j), s1 = s0 && i + 1 <= p.nx - 3;   // a pair lies in one cell
                const unsigned at = (unsigned)(j * p.pitch + i);
                if (s1) {
#pragma unroll
                    for (int k = 0; k < 9; ++k)
                        *reinterpret_cast<uint32_t *>((fout + (long long)k * p.plane) + at) = Pair2<T>::pack(o[k]);
                } else if (s0) {
#pragma unroll
                    for (int k = 0; k < 9; ++k) (fout + (long long)k * p.plane)[at] = Store<T>::pack(o[k].x);
                }
            }
            p0 = w[0]; p2b = p2; p2 = w[2]; q1 = c1; q3 = c3; q5b = q5; q5 = c5; q6b = q6; q6 = c6;
        }
    } else {
        C p0 = 0, p2 = 0, p2b = 0, q1 = 0, q3 = 0, q5 = 0, q5b = 0, q6 = 0, q6b = 0;
        for (int r = 0; r < nrows; ++r) {
            const int q = r % KS;
            ok = wait(&full[q], (uint32_t)((r / KS) & 1)) && ok;
            C g[9], o[9], rho, u, v;
            const T *b = buf + q * 9 * SEG + sh + col;
#pragma unroll
            for (int k = 0; k < 9; ++k) g[k] = b[k * SEG - lbm_ex(k)];
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[q]);
            collide_interior<C, CONS0>(a, g, false, C(0), C(0), o, rho, u, v);
            refill(r);
            if (!__all_sync(0xffffffffu, ok)) break;
            const C c1 = from_left(o[1]), c3 = from_right(o[3]), c5 = from_left(o[5]), c6 = from_right(o[6]);
            const C c7 = from_right(o[7]), c8 = from_left(o[8]);
            if (r > 1) {
                const int j = y0 - 2 + r;
                g[0] = p0; g[1] = q1; g[2] = p2b; g[3] = q3; g[4] = o[4]; g[5] = q5b; g[6] = q6b;
                g[7] = c7;
                g[8] = c8;
                C w[9];
                collide_interior<C, CONS0>(a, g, false, C(0), C(0), w, rho, u, v);
                if (out0 && !kept(i, j)) {
                    const unsigned at = (unsigned)(j * p.pitch + i);
#pragma unroll
                    for (int k = 0; k < 9; ++k) (fout + (long long)k * p.plane)[at] = w[k];
                }
            }
            p0 = o[0]; p2b = p2; p2 = o[2]; q1 = c1; q3 = c3; q5b = q5; q5 = c5; q6b = q6; q6 = c6;
        }
    }
    if (__syncthreads_or(!ok)) {
        // report, then wait (bounded) for this CTA's copies still in flight
        if (tid == 0) atomicOr(p.status, LBM_ST_TIMEOUT);
        for (int q = 0; q < KS; ++q) {
            int spins = 0;
            while (!mbar_try_wait(&full[q], 0) && !mbar_try_wait(&full[q], 1) && ++spins < (1 << 20)) {
            }
        }
    }
}

template <typename T, typename C, bool CONS0>
__global__ void __launch_bounds__(PT, sizeof(T) == 8 ? 2 : 4) kf_pair(const __grid_constant__ PairArgs<C> p)
{
    extern __shared__ __align__(128) unsigned char sm[];
    pair_cta<T, C, CONS0>(p, blockIdx.x, blockIdx.y, sm);
}

// ---- the nodes near a body and at the edge -----------------------------------

template <typename C> struct NearArgs {
    KFArgs<C> kf;                // of the step: fin, fout, the step's correction tiles
    const unsigned char *near;
    const int *list;             // the near cells
    const int *count;
    int cells_x, cells_y;
    int phase;                   // 0: first step (the cells and the nodes next to them), 1: second
};

template <typename C>
__device__ __forceinline__ bool near_tile(const KFArgs<C> &a, const PatchInfo &r, int i, int j)
{
    const unsigned li = (unsigned)(i - r.i0), lj = (unsigned)(j - r.j0);
    if (li >= (unsigned)r.w || lj >= (unsigned)r.h) return false;
    const unsigned tx = li >> 4, t = (lj >> 4) * (unsigned)a.tiles_x + tx;
    if (tx >= (unsigned)a.tiles_x || t >= (unsigned)a.tiles_n) {
        atomicOr(a.status, LBM_ST_INDEX_LATTICE);
        return false;
    }
    return a.tiles[(long long)t * a.tile_stride] > 0;
}

// one node of a step outside its correction tiles, by the arithmetic of the
// lattice kernels (with FP32 arithmetic the paired update, the node in both
// halves); neighbouring cells and the frame may take the same node, with the
// same result
template <typename T, typename C, bool CONS0>
__device__ __forceinline__ void near_node(const KFArgs<C> &a, const PatchInfo &pr, int i, int j)
{
    if (near_tile(a, pr, i, j)) return;
    const T *fin = (const T *)a.fin;
    C g[9], o[9], rho, u, v;
    if (i == 0 || i == a.nx - 1 || j == 0 || j == a.ny - 1) {
        edge_update<T, C>(a, fin, i, j, o, rho, u, v);
    } else {
        pull<T, C>(fin, a.plane, a.pitch, i, j, g);
        if constexpr (std::is_same<C, float>::value) {
            float2 gg[9], oo[9], r2, u2, v2;
#pragma unroll
            for (int k = 0; k < 9; ++k) gg[k] = make_float2(g[k], g[k]);
            collide_pair<CONS0, false>(a, gg, oo, r2, u2, v2);
#pragma unroll
            for (int k = 0; k < 9; ++k) o[k] = oo[k].x;
        } else {
            collide_interior<C, CONS0>(a, g, false, C(0), C(0), o, rho, u, v);
        }
    }
    store_node<T, C, false>(a, (T *)a.fout, i, j, o, rho, u, v);
}

// CTAs from the first on: the near cells, strided over the first `cell_ctas`
// of them; the CTAs after those: the nodes at the edge (phase 0: what their
// second step needs, twice the frame)
template <typename T, typename C, bool CONS0>
__device__ __forceinline__ void near_cta(const NearArgs<C> &n, int b, int cell_ctas, int all)
{
    const KFArgs<C> &a = n.kf;
    const PatchInfo pr = *a.pinfo;
    const int tid = threadIdx.x;
    if (b < cell_ctas) {
        const int cells = n.cells_x * n.cells_y;
        int count = *n.count;
        if (count < 0 || count > cells) {
            if (tid == 0) atomicOr(a.status, LBM_ST_INDEX_LATTICE);
            count = 0;
        }
        for (int c = b; c < count; c += cell_ctas) {
            const int cell = n.list[c];
            if (cell < 0 || cell >= cells) {
                if (tid == 0) atomicOr(a.status, LBM_ST_INDEX_LATTICE);
                continue;
            }
            const int ci = cell % n.cells_x * CELL, cj = cell / n.cells_x * CELL;
            const int i = ci + (tid & 15), j = cj + (tid >> 4);
            if (i < a.nx && j < a.ny) near_node<T, C, CONS0>(a, pr, i, j);
            // the nodes around the cell, where no near cell has them
            if (n.phase == 0 && tid < 4 * CELL + 4) {
                const int t = tid;
                const int ri = t < CELL + 2 ? ci - 1 + t : t < 2 * CELL + 4 ? ci - 1 + t - (CELL + 2)
                               : t < 3 * CELL + 4 ? ci - 1 : ci + CELL;
                const int rj = t < CELL + 2 ? cj - 1 : t < 2 * CELL + 4 ? cj + CELL
                               : t < 3 * CELL + 4 ? cj + t - (2 * CELL + 4) : cj + t - (3 * CELL + 4);
                if (ri >= 0 && rj >= 0 && ri < a.nx && rj < a.ny && !n.near[(rj >> 4) * n.cells_x + (ri >> 4)])
                    near_node<T, C, CONS0>(a, pr, ri, rj);
            }
        }
        return;
    }
    const int d = n.phase == 0 ? 2 * FRAME : FRAME;   // (lattices of kf_pair are wider than 4 d)
    const int rows = 2 * d * a.nx, total = rows + 2 * d * (a.ny - 2 * d);
    for (int e = (b - cell_ctas) * PT + tid; e < total; e += (all - cell_ctas) * PT) {
        int i, j;
        if (e < rows) {
            const int q = e / a.nx;
            i = e - q * a.nx;
            j = q < d ? q : a.ny - 2 * d + q;
        } else {
            const int q = (e - rows) % (2 * d);
            j = d + (e - rows) / (2 * d);
            i = q < d ? q : a.nx - 2 * d + q;
        }
        near_node<T, C, CONS0>(a, pr, i, j);
    }
}

template <typename T, typename C, bool CONS0>
__global__ void __launch_bounds__(PT) kf_near(const __grid_constant__ NearArgs<C> n, int cell_ctas)
{
    near_cta<T, C, CONS0>(n, blockIdx.x, cell_ctas, gridDim.x);
}

// The near cells of a pair of steps (e, e + 1), e even: the cells of the first
// step's correction tiles and of the nodes next to them, and of the second
// step's tiles. One CTA per pair of the factorization batch; geometry only,
// so part of its chain. `near`: a byte per cell, then `list` in cell order.
constexpr int NEAR_THREADS = 1024;
__device__ __forceinline__ void near_cells(const IBArgs &base, int e, int nx, int ny, unsigned char *near, int *list, int *count)
{
    __shared__ int wsum[NEAR_THREADS / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cx = (nx + CELL - 1) / CELL, cy = (ny + CELL - 1) / CELL, cells = cx * cy;
    for (int c = tid; c < cells; c += NEAR_THREADS) near[c] = 0;
    __syncthreads();
    for (int s = 0; s < 2; ++s) {
        const IBArgs a = lbm_ib::step_args(base, e + s);
        const PatchInfo pr = *a.pinfo;
        const int nt = lbm_ib::patch_tiles(a), grow = s == 0 ? 1 : 0;
        int ntile = *a.nsup;
        if (ntile < 0 || ntile > nt) {
            if (tid == 0) atomicOr(a.fstatus, LBM_ST_INDEX_LATTICE);
            ntile = 0;
        }
        for (int c = tid; c < ntile; c += NEAR_THREADS) {
            const int tile = a.ctile[c];
            if (tile < 0 || tile >= nt) {
                atomicOr(a.fstatus, LBM_ST_INDEX_LATTICE);
                continue;
            }
            const int x0 = pr.i0 + tile % a.tiles_x * TILE - grow, y0 = pr.j0 + tile / a.tiles_x * TILE - grow;
            const int x1 = x0 + TILE - 1 + 2 * grow, y1 = y0 + TILE - 1 + 2 * grow;
            for (int q = max(y0, 0) / CELL; q <= min(y1, ny - 1) / CELL; ++q)
                for (int p = max(x0, 0) / CELL; p <= min(x1, nx - 1) / CELL; ++p) near[q * cx + p] = 1;
        }
    }
    __syncthreads();
    const int per = (cells + NEAR_THREADS - 1) / NEAR_THREADS, c0 = min(cells, tid * per), c1 = min(cells, c0 + per);
    int n = 0;
    for (int c = c0; c < c1; ++c) n += near[c];
    int x = n;   // inclusive scan within the warp
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    int before = 0;
    for (int w = 0; w < warp; ++w) before += wsum[w];
    int pos = before + x - n;
    for (int c = c0; c < c1; ++c)
        if (near[c]) list[pos++] = c;
    if (tid == NEAR_THREADS - 1) *count = before + x;
}

__global__ void __launch_bounds__(NEAR_THREADS) ib_near(const IBArgs base, int e0, unsigned char *near, int *list, int *count,
                                                        int cells, int cap)
{
    const int e = e0 + 2 * (int)blockIdx.x, slot = e / 2 % (base.nslots / 2);
    near_cells(base, e, base.nx, base.ny, near + (long long)slot * cap, list + (long long)slot * cells, count + slot);
}

int cells_of(const lbm_handle *h, int *cx, int *cy)
{
    *cx = (h->nx + CELL - 1) / CELL;
    *cy = (h->ny + CELL - 1) / CELL;
    return *cx * *cy;
}

// rows a CTA writes. Two more are computed by it for the first step only, so
// the kernel alone is fastest with 16 to 20; but the immersed-boundary kernels
// beside it start as its CTAs leave, and the step as a whole is faster with
// shorter ones (4096x2048, us a step with 8, 10, 12, 14, 20 rows: FP32 72.7,
// 72.4, 72.6, 72.1, 75.0; FP16 62.1, 61.2, 60.8, 62.6, 62.1; FP64, by an
// earlier form, 133.6, 130.3, 129.3, 128.3, 127.5). Fewer where the lattice
// has not two waves of such CTAs.
template <typename T> int pair_rows(const lbm_handle *h)
{
    const int per_sm = sizeof(T) == 8 ? 2 : 4, strips = (h->nx - 2 * FRAME + pair_out<T>() - 1) / pair_out<T>();
    int r = sizeof(T) == 8 ? 20 : 12;
    while (r > 8 && strips * ((h->ny - 2 * FRAME + r - 1) / r) < 2 * 148 * per_sm) r -= 2;
    return r;
}

template <typename T, typename C>
PairArgs<C> pair_args(const lbm_handle *h, const void *fin, void *fout, int step)
{
    PairArgs<C> p;
    int cx, cy;
    const int cells = cells_of(h, &cx, &cy);
    const KFArgs<C> k = make_kf_args<C>(const_cast<lbm_handle *>(h), fin, fout, nullptr, KF_ALL);
    p.fin = fin;
    p.fout = fout;
    p.nx = h->nx;
    p.ny = h->ny;
    p.pitch = h->pitch;
    p.plane = h->plane;
    for (int q = 0; q < 9; ++q) { p.s[q] = k.s[q]; p.sc[q] = k.sc[q]; }
    p.rows = pair_rows<T>(h);
    p.near = h->d_near + (size_t)(step / 2 % (h->nslots / 2)) * near_bytes(cells);
    p.cells_x = cx;
    p.status = h->d_status;
    return p;
}

template <typename T, typename C, bool CONS0>
int launch_pair_t(lbm_handle *h, const void *fin, void *fout, cudaStream_t st)
{
    const PairArgs<C> p = pair_args<T, C>(h, fin, fout, h->n);
    auto kernel = kf_pair<T, C, CONS0>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pair_smem<T>()) != cudaSuccess) return -1;
    const dim3 grid((h->nx - 2 * FRAME + pair_out<T>() - 1) / pair_out<T>(), (h->ny - 2 * FRAME + p.rows - 1) / p.rows);
    kernel<<<grid, PT, pair_smem<T>(), st>>>(p);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

template <typename T, typename C, bool CONS0>
int launch_near_t(lbm_handle *h, const void *fin, void *fout, int step, int phase, cudaStream_t st)
{
    NearArgs<C> n;
    const int cells = cells_of(h, &n.cells_x, &n.cells_y), slot = step / 2 % (h->nslots / 2);
    n.kf = make_kf_args<C>(h, fin, fout, nullptr, KF_OUTER);
    n.near = h->d_near + (size_t)slot * near_bytes(cells);
    n.list = h->d_near_list + (size_t)slot * cells;
    n.count = h->d_near_count + slot;
    n.phase = phase;
    // (a contour of 1024 markers on a chord of 512 has some 450 near cells)
    const int cell_ctas = std::min(cells, 2 * 148), edge_ctas = 24;
    kf_near<T, C, CONS0><<<cell_ctas + edge_ctas, PT, 0, st>>>(n, cell_ctas);
    h->count(0, 1);   // (a part of the lattice)
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

bool zero_rates(const lbm_handle *h) { return h->s[0] == 0.0 && h->s[3] == 0.0 && h->s[5] == 0.0; }

}  // namespace

size_t near_bytes(int cells) { return ((size_t)cells + 255) / 256 * 256; }
int near_cells_of(const lbm_handle *h)
{
    int cx, cy;
    return cells_of(h, &cx, &cy);
}

// the near cells of the pairs of steps within step0 .. step0 + count - 1
int launch_near_cells(lbm_handle *h, int step0, int count, cudaStream_t st)
{
    const int e0 = (step0 + 1) / 2 * 2, pairs = (step0 + count - e0) / 2;
    if (pairs <= 0) return 0;
    IBArgs a;
    ib_args_write(h, nullptr, 0, &a);
    const int cells = near_cells_of(h);
    ib_near<<<pairs, NEAR_THREADS, 0, st>>>(a, e0, h->d_near, h->d_near_list, h->d_near_count, cells, (int)near_bytes(cells));
    h->count(0, 1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// both steps h->n, h->n + 1 (h->n even) of the nodes away from bodies and edge
int launch_pair(lbm_handle *h, const void *fin, void *fout, cudaStream_t st)
{
    const bool c0 = zero_rates(h);
    switch (h->prec) {
    case LBM_PREC_FP32: return c0 ? launch_pair_t<float, float, true>(h, fin, fout, st) : launch_pair_t<float, float, false>(h, fin, fout, st);
    case LBM_PREC_FP64: return c0 ? launch_pair_t<double, double, true>(h, fin, fout, st) : launch_pair_t<double, double, false>(h, fin, fout, st);
    case LBM_PREC_FP16: return c0 ? launch_pair_t<__half, float, true>(h, fin, fout, st) : launch_pair_t<__half, float, false>(h, fin, fout, st);
    case LBM_PREC_BF16: return c0 ? launch_pair_t<__nv_bfloat16, float, true>(h, fin, fout, st) : launch_pair_t<__nv_bfloat16, float, false>(h, fin, fout, st);
    }
    return -1;
}

// one of the two steps of the other nodes, except the step's correction tiles
// (h->pinfo_slot: the step's slot); `step`: the pair's first
int launch_near(lbm_handle *h, const void *fin, void *fout, int step, int phase, cudaStream_t st)
{
    const bool c0 = zero_rates(h);
    switch (h->prec) {
    case LBM_PREC_FP32: return c0 ? launch_near_t<float, float, true>(h, fin, fout, step, phase, st) : launch_near_t<float, float, false>(h, fin, fout, step, phase, st);
    case LBM_PREC_FP64: return c0 ? launch_near_t<double, double, true>(h, fin, fout, step, phase, st) : launch_near_t<double, double, false>(h, fin, fout, step, phase, st);
    case LBM_PREC_FP16: return c0 ? launch_near_t<__half, float, true>(h, fin, fout, step, phase, st) : launch_near_t<__half, float, false>(h, fin, fout, step, phase, st);
    case LBM_PREC_BF16: return c0 ? launch_near_t<__nv_bfloat16, float, true>(h, fin, fout, step, phase, st) : launch_near_t<__nv_bfloat16, float, false>(h, fin, fout, step, phase, st);
    }
    return -1;
}
