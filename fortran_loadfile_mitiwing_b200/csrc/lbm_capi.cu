// lbm_capi.cu -- the extern "C" boundary (include/lbm_b200.h): handle
// lifetime, device memory, initial state, and the per-step launch sequence.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <type_traits>
#include <unordered_map>
#include <vector>

#include "lbm_internal.h"

namespace {

const double kWref[9] = {4.0 / 9.0, 1.0 / 9.0, 1.0 / 9.0, 1.0 / 9.0, 1.0 / 9.0,
                         1.0 / 36.0, 1.0 / 36.0, 1.0 / 36.0, 1.0 / 36.0};
const int kEx[9] = {0, 1, 0, -1, 0, 1, -1, -1, 1};
const int kEy[9] = {0, 0, 1, 0, -1, 1, 1, -1, -1};
const int kRing = 2048;   // force rows kept on the device between host copies
const int kLoopSpare = 16;   // SMs left free beside a step_loop launch


int set_err(lbm_handle *h, int code, const char *msg)
{
    if (h) h->err = msg;
    return code;
}

int cuda_err(lbm_handle *h, cudaError_t e, const char *where)
{
    char buf[256];
    snprintf(buf, sizeof buf, "%s: %s", where, cudaGetErrorString(e));
    return set_err(h, LBM_ERR_CUDA, buf);
}

#define CK(call, where)                                   \
    do {                                                  \
        cudaError_t e_ = (call);                          \
        if (e_ != cudaSuccess) return cuda_err(h, e_, where); \
    } while (0)

size_t compute_size(int prec) { return prec == LBM_PREC_FP64 ? sizeof(double) : sizeof(float); }

size_t storage_size(int prec)
{
    switch (prec) {
    case LBM_PREC_FP64: return 8;
    case LBM_PREC_FP32: return 4;
    default: return 2;
    }
}

// single-precision lattice weights of D2Q9model (D2Q9model.f90:24-32)
double wsingle(int k) { return k == 0 ? (double)(4.0f / 9.0f) : (k < 5 ? (double)(1.0f / 9.0f) : (double)(1.0f / 36.0f)); }

// D2Q9feq (D2Q9model.f90:35-46), host FP64
double feq(double rh, double u1, double v1, int k)
{
    const double eu = (double)kEx[k] * u1 + (double)kEy[k] * v1;
    const double utwo = u1 * u1 + v1 * v1;
    return wsingle(k) * rh * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * utwo);
}

// device allocations of the handles, owner and size (lbm_device_bytes)
std::mutex g_alloc_mu;
std::unordered_map<void *, std::pair<lbm_handle *, size_t>> g_allocs;

// The handles' device memory comes from one stream-ordered memory pool per
// device, owned by the library, that keeps what freed handles return
// (release threshold: never) for the next allocations: a handle created
// after another was destroyed, as a sweep or a serving loop does many times,
// reuses memory that is already mapped instead of mapping it again, and a
// free does not synchronise the device as cudaFree does. The pool holds the
// process's peak of live handle memory until the process exits.
cudaMemPool_t handle_pool(int dev)
{
    static std::mutex mu;
    static std::unordered_map<int, cudaMemPool_t> pools;
    std::lock_guard<std::mutex> lock(mu);
    auto it = pools.find(dev);
    if (it != pools.end()) return it->second;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
        cudaGetLastError();
        pool = nullptr;   // plain cudaMalloc / cudaFree then
    } else {
        unsigned long long keep = ~0ull;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    pools[dev] = pool;
    return pool;
}

// allocations from the pool, by address (freed back to it)
std::unordered_map<void *, bool> g_pooled;

// Every allocation is zero-filled on the handle's stream, ahead of all work
// that uses it (the other streams are ordered after the main stream's
// position by events or a synchronisation), so that no kernel can see data a
// freed allocation of an earlier handle left in the same memory.
template <typename P> cudaError_t dmalloc(lbm_handle *h, P **p, size_t bytes)
{
    void *q = nullptr;
    cudaMemPool_t pool = h->stream ? handle_pool(h->dev) : nullptr;
    cudaError_t e = cudaErrorMemoryAllocation;
    if (pool && (e = cudaMallocFromPoolAsync(&q, bytes, pool, h->stream)) != cudaSuccess) {
        // a pool unusable here (a context other than the one it was made in,
        // or one reset since): a plain allocation
        cudaGetLastError();
        pool = nullptr;
    }
    if (!pool) e = cudaMalloc(&q, bytes);
    if (e != cudaSuccess) return e;
    e = h->stream ? cudaMemsetAsync(q, 0, bytes, h->stream) : cudaMemset(q, 0, bytes);
    if (e != cudaSuccess) {
        if (pool)
            cudaFreeAsync(q, h->stream);
        else
            cudaFree(q);
        return e;
    }
    if (pool) {
        std::lock_guard<std::mutex> lock(g_alloc_mu);
        g_pooled[q] = true;
    }
    *p = (P *)q;
    std::lock_guard<std::mutex> lock(g_alloc_mu);
    g_allocs[q] = {h, bytes};
    h->dev_bytes += (long long)bytes;
    return e;
}

// Callers first synchronise the streams of the handle that owns p (no queued
// work may still use it); a pooled allocation goes back to the pool on the
// owner's main stream, idle by then.
void free_dev(void *&p)
{
    if (p) {
        bool pooled = false;
        cudaStream_t st = nullptr;
        {
            std::lock_guard<std::mutex> lock(g_alloc_mu);
            auto it = g_allocs.find(p);
            if (it != g_allocs.end()) {
                it->second.first->dev_bytes -= (long long)it->second.second;
                st = it->second.first->stream;
                g_allocs.erase(it);
            }
            auto jt = g_pooled.find(p);
            if (jt != g_pooled.end()) {
                pooled = true;
                g_pooled.erase(jt);
            }
        }
        if (pooled)
            cudaFreeAsync(p, st);
        else
            cudaFree(p);
    }
    p = nullptr;
}
template <typename P> void free_devp(P *&p)
{
    void *q = (void *)p;
    free_dev(q);
    p = nullptr;
}

// waits for all of the handle's queued work (lattice, immersed-boundary,
// check and factorization streams): before its device buffers are rewritten
// or freed
void quiesce(lbm_handle *h)
{
    if (h->fstream) cudaStreamSynchronize(h->fstream);
    if (h->side) cudaStreamSynchronize(h->side);
    if (h->cstream) cudaStreamSynchronize(h->cstream);
    if (h->nstream) cudaStreamSynchronize(h->nstream);
    if (h->stream) cudaStreamSynchronize(h->stream);
}

// rows of the motion step table (mode.f90:176-269), host FP64
void lookup_row(const std::vector<double> &tab, int rows, int cols, double t, int &idx, double *row)
{
    auto T = [&](int r, int c) { return tab[(size_t)c * rows + r]; };
    if (t <= T(0, 0)) {
        idx = 0;
        for (int c = 0; c < cols; ++c) row[c] = T(0, c);
        row[0] = t;
        return;
    }
    if (t >= T(rows - 1, 0)) {
        idx = std::max(rows - 2, 0);
        for (int c = 0; c < cols; ++c) row[c] = T(rows - 1, c);
        row[0] = t;
        return;
    }
    int mi = std::max(0, std::min(idx, rows - 2));
    while (mi > 0 && t < T(mi, 0)) mi--;
    while (mi < rows - 2 && t > T(mi + 1, 0)) mi++;
    idx = mi;
    if (fabs(t - T(mi, 0)) <= 1.0e-12) {
        for (int c = 0; c < cols; ++c) row[c] = T(mi, c);
        row[0] = t;
        return;
    }
    if (fabs(t - T(mi + 1, 0)) <= 1.0e-12) {
        for (int c = 0; c < cols; ++c) row[c] = T(mi + 1, c);
        row[0] = t;
        return;
    }
    const double t1 = T(mi, 0), t2 = T(mi + 1, 0);
    if (fabs(t2 - t1) <= 1.0e-14) {
        for (int c = 0; c < cols; ++c) row[c] = T(mi, c);
        row[0] = t;
        return;
    }
    const double weight = (t - t1) / (t2 - t1);
    for (int c = 0; c < cols; ++c) row[c] = (1.0 - weight) * T(mi, c) + weight * T(mi + 1, c);
    row[0] = t;
}

// releases the immersed-boundary scratch (sizes depend on geometry and motion)
void free_ib(lbm_handle *h)
{
    if (h->fstream) cudaStreamSynchronize(h->fstream);
    if (h->side) cudaStreamSynchronize(h->side);
    if (h->cstream) cudaStreamSynchronize(h->cstream);
    if (h->nstream) cudaStreamSynchronize(h->nstream);
    if (h->stream) cudaStreamSynchronize(h->stream);
    h->ib_ready = 0;
    forget_batches(h);
    free_devp(h->d_mk); free_devp(h->d_rhs); free_devp(h->d_B); free_devp(h->d_y); free_devp(h->d_partial);
    free_devp(h->d_bD); free_devp(h->d_bL); free_devp(h->d_gf); free_devp(h->d_fmode); free_devp(h->d_fstatus); free_devp(h->d_tiles); free_devp(h->d_nsup); free_devp(h->d_ctile);
    free_dev(h->fmid_alloc); h->fmid = nullptr; h->pairs = 0;
    free_devp(h->d_near); free_devp(h->d_near_list); free_devp(h->d_near_count);
    free_devp(h->d_perm); free_devp(h->d_key); free_devp(h->d_reach); free_devp(h->d_wmax);
}

// Whether a handle's steps run two at a time: lattices that step_loop does not
// take, of 40 MB of traffic a step or more. Below, where the flow chain is the
// step, the two forms differ by no more than the runs do, and the state between
// the steps would take half as much memory again. us a step, one and two at a
// time, 580 markers: FP32 15 MB 34 and 34, 30 MB 39 and 35, 40 MB 41 and 33, 80
// MB 39 and 37, 120 MB 49 and 37; FP16 30 MB 39 and 34, 40 MB 34 and 33, 80 MB 45
// and 37; FP64 30 MB 33 and 33, 40 MB 34 and 33, 80 MB 34 and 36, 120 MB 46 and 37.
bool pairs_fit(const lbm_handle *h)
{
    return h->overlap && h->kf_tma && h->nseg > 0 && h->nslots % 2 == 0 && h->fbatch % 2 == 0 && !loop_fits(h) && h->nx >= 64 &&
           h->ny >= 64 && h->plane < (1ll << 31) && 18ll * h->elem * h->plane >= 40000000ll;
}

// Whether some step of the motion may need the dense factor of the marker
// system: a coupling of more than kBand places in the solve order (ib_factor),
// that is two markers whose support boxes (at most 5 lattice units from first
// to last node) share a node with kBand others or more between them. The
// factor takes 8 nseg^2 bytes a step slot and next to no case uses it (a
// contour with a marker per lattice unit has couplings of some 14 places), so
// it is allocated only where this bound does not rule it out.
constexpr int kBand = 16;
constexpr double kSpan = 5.0 + 1.0e-6;   // lattice units; positions are rounded

// The solve order of one rigid body, kept for the whole run: by body-frame
// chordwise position (two markers whose support boxes overlap are less than
// 5 sqrt(2) lattice units apart in any orientation). key: the positions.
void body_order(const lbm_handle *h, std::vector<int> &perm, std::vector<double> &key)
{
    const int n = h->nseg;
    std::vector<double> x(n);
    perm.resize(n);
    key.resize(n);
    for (int k = 0; k < n; ++k) {
        perm[k] = k;
        x[k] = 0.5 * (h->hx0[k] + h->hx0[k + 1]);
    }
    std::stable_sort(perm.begin(), perm.end(), [&](int p, int q) { return x[p] < x[q]; });
    for (int q = 0; q < n; ++q) key[q] = x[perm[q]];
}

// One body in its order
bool band_exceeded(const lbm_handle *h, const std::vector<int> &perm, const std::vector<double> &key)
{
    const int n = h->nseg;
    const double reach = sqrt(2.0) * kSpan * h->p.scale;
    auto y = [&](int q) { return 0.5 * (h->hy0[perm[q]] + h->hy0[perm[q] + 1]); };
    for (int p = 0; p < n; ++p)
        for (int q = p + kBand + 1; q < n && key[q] - key[p] <= reach; ++q)
            if (hypot(key[q] - key[p], y(q) - y(p)) <= reach) return true;
    return false;
}

// What the rows of a step table span: angles, and displacements (x, y) of body
// q less those of body p < q
struct MotionRange {
    double a0[LBM_MAXW], a1[LBM_MAXW], c0[2][LBM_MAXW][LBM_MAXW], c1[2][LBM_MAXW][LBM_MAXW];
    MotionRange()
    {
        std::fill(a0, a0 + LBM_MAXW, 1e300);
        std::fill(a1, a1 + LBM_MAXW, -1e300);
        std::fill(&c0[0][0][0], &c0[0][0][0] + 2 * LBM_MAXW * LBM_MAXW, 1e300);
        std::fill(&c1[0][0][0], &c1[0][0][0] + 2 * LBM_MAXW * LBM_MAXW, -1e300);
    }
    void add(const double *row, int nwing)
    {
        for (int p = 0; p < nwing; ++p) {
            const double a = row[1 + 9 * p];
            a0[p] = a < a0[p] ? a : a0[p];
            a1[p] = a > a1[p] ? a : a1[p];
            for (int d = 0; d < 2; ++d)
                for (int q = p + 1; q < nwing; ++q) {
                    const double c = row[4 + 3 * d + 9 * q] - row[4 + 3 * d + 9 * p];
                    c0[d][p][q] = c < c0[d][p][q] ? c : c0[d][p][q];
                    c1[d][p][q] = c > c1[d][p][q] ? c : c1[d][p][q];
                }
        }
    }
};

// A body of several, over the angles of its motion
struct BodyRange {
    std::vector<double> x, y;    // markers in the body's frame, lattice units
    double a0 = 1e300, a1 = -1e300, r = 0.0;   // angles, distance of the farthest marker
    double lo[2], hi[2];         // extent along x and y about the pivot, over all angles,
    double in_lo[2], in_hi[2];   // and what it covers at every angle
    // samples of the angle between the nearest of which and any other angle no
    // marker moves more than `move` relative to another
    double samples(double move) const { return std::ceil(r * (a1 - a0) / move) + 1.0; }
    // positions along an axis, f(position) for each marker of sample t of n
    template <class F> void each(int t, int n, int d, F f) const
    {
        const double a = n > 1 ? a0 + (a1 - a0) * t / (n - 1) : a0, ca = cos(a), sn = d == 0 ? sin(a) : -sin(a);
        const double *p = d == 0 ? x.data() : y.data(), *q = d == 0 ? y.data() : x.data();
        for (size_t k = 0; k < x.size(); ++k) f(ca * p[k] + sn * q[k]);
    }
    void extents()
    {
        const double move = std::max(1.0, r * (a1 - a0) / 15.0);
        const int n = (int)samples(move);
        for (int d = 0; d < 2; ++d) {
            lo[d] = in_hi[d] = 1e300;
            hi[d] = in_lo[d] = -1e300;
            for (int t = 0; t < n; ++t) {
                double v0 = 1e300, v1 = -1e300;
                each(t, n, d, [&](double v) {
                    v0 = v < v0 ? v : v0;
                    v1 = v > v1 ? v : v1;
                });
                lo[d] = std::min(lo[d], v0 - move);
                hi[d] = std::max(hi[d], v1 + move);
                in_lo[d] = std::max(in_lo[d], v0 + move);
                in_hi[d] = std::min(in_hi[d], v1 - move);
            }
        }
    }
    // a bound on the markers within kSpan along an axis: those of 13 successive
    // bins of half a unit, which hold any window of kSpan + kMove
    static constexpr double kMove = 0.9;
    int most(int d) const
    {
        std::vector<int> bin((size_t)(4.0 * r) + 16);
        const int n = (int)samples(kMove);
        int m = 0;
        for (int t = 0; t < n; ++t) {
            std::fill(bin.begin(), bin.end(), 0);
            each(t, n, d, [&](double v) { ++bin[(size_t)(2.0 * (v + r) + 1.0)]; });   // |v| <= r, but for rounding
            int sum = 0;
            for (size_t q = 0; q < bin.size(); ++q) {
                sum += bin[q] - (q >= 13 ? bin[q - 13] : 0);
                m = std::max(m, sum);
            }
        }
        return m;
    }
    bool same(const BodyRange &o) const { return x == o.x && y == o.y && a0 == o.a0 && a1 == o.a1; }
};

// Several bodies: the order follows the longer axis of all markers; a coupling
// spans no more places than a window of kSpan along it holds markers, of the
// bodies that can be in it together.
bool window_exceeded(const lbm_handle *h, const MotionRange &range)
{
    const int nw = h->nwing;
    std::vector<BodyRange> body(nw);
    for (int w = 0; w < nw; ++w)
        for (int k = 0; k < h->spw; ++k) {
            const int q = w * h->ppw + k;
            body[w].x.push_back(0.5 * (h->hx0[q] + h->hx0[q + 1]) / h->p.scale);
            body[w].y.push_back(0.5 * (h->hy0[q] + h->hy0[q + 1]) / h->p.scale);
        }
    for (int w = 0; w < nw; ++w) {
        body[w].a0 = range.a0[w];
        body[w].a1 = range.a1[w];
    }
    for (BodyRange &b : body) {
        for (size_t k = 0; k < b.x.size(); ++k) b.r = std::max(b.r, hypot(b.x[k], b.y[k]));
        const double n = b.samples(BodyRange::kMove);
        if (!(n >= 1.0 && n <= 1000.0 && b.r <= 1.0e5)) return true;   // (turns of a large body: not worth the time)
        b.extents();
    }
    double cloud_min[2] = {0.0, 0.0}, cloud_max[2] = {0.0, 0.0};   // extent of all markers
    double c0[2][LBM_MAXW][LBM_MAXW], c1[2][LBM_MAXW][LBM_MAXW];   // from pivot p to pivot q, lattice units
    for (int d = 0; d < 2; ++d)
        for (int p = 0; p < nw; ++p)
            for (int q = 0; q < nw; ++q) {
                c0[d][p][q] = (q > p ? range.c0[d][p][q] : q < p ? -range.c1[d][q][p] : 0.0) / h->p.scale;
                c1[d][p][q] = (q > p ? range.c1[d][p][q] : q < p ? -range.c0[d][q][p] : 0.0) / h->p.scale;
                cloud_min[d] = std::max(cloud_min[d], c0[d][p][q] + body[q].in_hi[d] - body[p].in_lo[d]);
                cloud_max[d] = std::max(cloud_max[d], c1[d][p][q] + body[q].hi[d] - body[p].lo[d]);
            }
    for (int d = 0; d < 2; ++d) {
        if (cloud_max[d] < cloud_min[d ^ 1]) continue;   // never the longer axis
        std::vector<int> most(nw);
        for (int p = 0; p < nw; ++p) {
            int q = 0;
            while (q < p && !body[q].same(body[p])) ++q;
            most[p] = q < p ? most[q] : body[p].most(d);
        }
        for (int p = 0; p < nw; ++p) {
            int window = 0;
            for (int q = 0; q < nw; ++q)
                if (c0[d][p][q] + body[q].lo[d] - body[p].hi[d] <= kSpan && body[p].lo[d] - c1[d][p][q] - body[q].hi[d] <= kSpan)
                    window += most[q];
            if (window > kBand + 1) return true;
        }
    }
    return false;
}

// Allocates the immersed-boundary scratch once geometry and motion are known:
// the correction patch is sized by the largest per-step rectangle of the
// bodies' bounding discs over the whole motion table.
int ensure_ib(lbm_handle *h)
{
    if (h->ib_ready) return LBM_OK;
    int wmax = 0, hmax = 0;
    MotionRange range;
    double gx0 = 1e300, gx1 = -1e300, gy0 = 1e300, gy1 = -1e300;   // motion envelope (lattice units)
    if (h->nseg > 0) {
        std::vector<double> R(h->nwing, 0.0);
        for (int w = 0; w < h->nwing; ++w)
            for (int p = 0; p < h->ppw; ++p) {
                const double x = h->hx0[w * h->ppw + p], y = h->hy0[w * h->ppw + p];
                R[w] = std::max(R[w], sqrt(x * x + y * y));
            }
        for (double &r : R) r = r / h->p.scale + 4.0;
        const double *T = h->mstep_host.data();
        const int nw = h->nwing, cols = h->mcols;
        const double scale = h->p.scale, xc = h->p.xc, yc = h->p.yc, ox = h->p.ox, oy = h->p.oy;
        auto rows = [&](auto several) {
            for (int s = 0; s < h->msteps; ++s) {
                const double *row = T + (size_t)s * cols;
                if constexpr (several) range.add(row, nw);
                double xlo = 1e300, xhi = -1e300, ylo = 1e300, yhi = -1e300;
                for (int w = 0; w < nw; ++w) {
                    const double sa = row[4 + 9 * w], sb = row[7 + 9 * w];
                    const double cx = (sa + xc - ox) / scale, cy = (sb + yc - oy) / scale, r = R[w];
                    xlo = std::min(xlo, cx - r); xhi = std::max(xhi, cx + r);
                    ylo = std::min(ylo, cy - r); yhi = std::max(yhi, cy + r);
                }
                wmax = std::max(wmax, (int)ceil(xhi - xlo) + 2);
                hmax = std::max(hmax, (int)ceil(yhi - ylo) + 2);
                gx0 = std::min(gx0, xlo); gx1 = std::max(gx1, xhi);
                gy0 = std::min(gy0, ylo); gy1 = std::max(gy1, yhi);
            }
        };
        if (nw > 1) rows(std::true_type());
        else rows(std::false_type());
        wmax = std::min(wmax, h->nx);
        hmax = std::min(hmax, h->ny);
    }
    h->patch_wmax = wmax;
    h->patch_hmax = hmax;
    // split rectangle: every support node of every step lies inside it (the
    // disc of radius R+4 lu around each pivot covers the marker boxes); x
    // bounds rounded out to multiples of 4, clipped to the interior
    h->env_x0 = h->env_y0 = h->env_w = h->env_h = 0;
    if (h->nseg > 0) {
        int x0 = std::max(4, ((int)floor(gx0) - 1) / 4 * 4), x1 = std::min(h->nx - 4, ((int)ceil(gx1) + 2 + 3) / 4 * 4);
        int y0 = std::max(1, (int)floor(gy0) - 1), y1 = std::min(h->ny - 1, (int)ceil(gy1) + 2);
        if (x1 > x0 && y1 > y0) { h->env_x0 = x0; h->env_y0 = y0; h->env_w = x1 - x0; h->env_h = y1 - y0; }
    }
    const int ns = std::max(1, h->nseg);
    const size_t S = (size_t)h->nslots, K = (size_t)h->fbatch;
    CK(dmalloc(h, &h->d_mk, S * sizeof(Marker) * ns), "alloc markers");
    CK(dmalloc(h, &h->d_rhs, S * sizeof(double) * 2 * ns), "alloc rhs");
    CK(dmalloc(h, &h->d_y, S * sizeof(double) * 2 * ns), "alloc y");
    std::vector<int> perm;
    std::vector<double> key;
    h->static_order = h->nwing == 1;
    if (h->static_order) body_order(h, perm, key);
    if (h->nseg > 0 && ((h->p.flags & LBM_FLAG_DENSE_SOLVE) ||
                        (h->nseg > kBand + 1 && (h->static_order ? band_exceeded(h, perm, key) : window_exceeded(h, range)))))
        CK(dmalloc(h, &h->d_B, S * sizeof(double) * (size_t)ns * ns), "alloc B");
    ib_factor_scratch(ns, &h->work_blocks, &h->gf_slot);
    CK(dmalloc(h, &h->d_bD, K * sizeof(double) * h->work_blocks), "alloc block D");
    CK(dmalloc(h, &h->d_bL, K * sizeof(double) * h->work_blocks), "alloc block L");
    CK(dmalloc(h, &h->d_gf, S * sizeof(double) * h->gf_slot), "alloc factor blocks");
    CK(dmalloc(h, &h->d_fmode, S * 2 * sizeof(int)), "alloc factor mode");
    CK(dmalloc(h, &h->d_fstatus, S * sizeof(unsigned)), "alloc factor status");
    CK(cudaMemsetAsync(h->d_fmode, 0, S * 2 * sizeof(int), h->stream), "clear factor mode");
    CK(cudaMemsetAsync(h->d_fstatus, 0, S * sizeof(unsigned), h->stream), "clear factor status");
    const int nblk = h->patch_gx() * h->patch_gy();
    // partials of the spread (per patch tile), of the residual check (per 8
    // markers) and the check's counter, per slot
    const size_t npart = (size_t)ib_partials_per_block() * nblk + 2 * (size_t)((ns + 7) / 8) + 1;
    h->part_stride = npart;
    CK(dmalloc(h, &h->d_partial, S * sizeof(double) * npart), "alloc partials");
    h->tiles_slot = (size_t)ib_tile_ints() * nblk;
    CK(dmalloc(h, &h->d_tiles, S * sizeof(int) * h->tiles_slot), "alloc tile lists");
    CK(cudaMemsetAsync(h->d_tiles, 0, S * sizeof(int) * h->tiles_slot, h->stream), "clear tile lists");
    CK(dmalloc(h, &h->d_nsup, S * sizeof(int)), "alloc tile counts");
    CK(dmalloc(h, &h->d_ctile, S * sizeof(int) * (size_t)nblk), "alloc correction tiles");
    CK(cudaMemsetAsync(h->d_nsup, 0, S * sizeof(int), h->stream), "clear tile counts");
    // solve order of the markers: one rigid body keeps its own; several are
    // sorted on the device every step
    CK(dmalloc(h, &h->d_perm, S * sizeof(int) * ns), "alloc perm");
    CK(dmalloc(h, &h->d_key, S * sizeof(double) * ns), "alloc key");
    CK(dmalloc(h, &h->d_reach, sizeof(double)), "alloc reach");
    CK(dmalloc(h, &h->d_wmax, K * sizeof(int)), "alloc wmax");
    CK(cudaMemsetAsync(h->d_wmax, 0, K * sizeof(int), h->stream), "clear wmax");
    if (h->static_order) {
        const double reach = 7.1 * h->p.scale;
        CK(cudaMemcpyAsync(h->d_perm, perm.data(), sizeof(int) * h->nseg, cudaMemcpyHostToDevice, h->stream), "copy perm");
        CK(cudaMemcpyAsync(h->d_key, key.data(), sizeof(double) * h->nseg, cudaMemcpyHostToDevice, h->stream), "copy key");
        CK(cudaMemcpyAsync(h->d_reach, &reach, sizeof(double), cudaMemcpyHostToDevice, h->stream), "copy reach");
        CK(cudaStreamSynchronize(h->stream), "sync order");
    }
    if (pairs_fit(h)) {
        const int cells = near_cells_of(h);
        if (!h->nstream) {   // with the events only here, most handles do without
            int low = 0, high = 0;
            cudaDeviceGetStreamPriorityRange(&low, &high);
            for (cudaEvent_t &ev : h->ev_near)
                if (!ev) CK(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming), "event");
            CK(cudaStreamCreateWithPriority(&h->nstream, cudaStreamNonBlocking, high), "near stream");
        }
        CK(dmalloc(h, &h->fmid_alloc, h->elem * (9 * (size_t)h->plane + 2 * LBM_FPAD)), "alloc f between");
        h->fmid = (char *)h->fmid_alloc + h->elem * LBM_FPAD;
        CK(dmalloc(h, &h->d_near, S / 2 * near_bytes(cells)), "alloc near cells");
        CK(dmalloc(h, &h->d_near_list, S / 2 * sizeof(int) * (size_t)cells), "alloc near list");
        CK(dmalloc(h, &h->d_near_count, S / 2 * sizeof(int)), "alloc near counts");
        h->pairs = 1;
    }
    if (ib_configure(h) != 0) return set_err(h, LBM_ERR_CUDA, "ib_configure failed");
    h->ib_ready = 1;
    return LBM_OK;
}

}  // namespace

// The error code and message of a device status word (the LBM_ST_* bits the
// kernels set); LBM_OK and "" for 0. An index error is reported first: the
// kernel that saw it skipped the access, so the step's results are not valid.
int status_error(unsigned st, std::string &msg)
{
    msg.clear();
    if (!st) return LBM_OK;
    if (st & LBM_ST_INDEX_MASK) {
        static const struct {
            unsigned bit;
            const char *kernel;
        } names[] = {{LBM_ST_INDEX_INTERP, "ib_interp"},     {LBM_ST_INDEX_ASSEMBLE, "ib_assemble"},
                     {LBM_ST_INDEX_FACTOR, "ib_factor"},     {LBM_ST_INDEX_SOLVE, "ib_solve"},
                     {LBM_ST_INDEX_SCATTER, "ib_tile_scatter"}, {LBM_ST_INDEX_SORT, "ib_tile_sort"},
                     {LBM_ST_INDEX_TILE, "ib_tile_update"}, {LBM_ST_INDEX_FORCES, "ib_forces"},
                     {LBM_ST_INDEX_RESIDUAL, "ib_residual"}, {LBM_ST_INDEX_LATTICE, "kf_tma"}};
        msg = "device index out of range, access skipped in:";
        for (const auto &n : names)
            if (st & n.bit) msg += std::string(" ") + n.kernel;
        return LBM_ERR_INDEX;
    }
    if (st & LBM_ST_TIMEOUT) {
        msg = "a bounded wait on the device gave up: for a shared-memory copy, or of a step_loop CTA for another";
        return LBM_ERR_CUDA;
    }
    if (st & LBM_ST_RANGE) {
        msg = "move_boundary: a marker support box reaches the three outermost node layers";
        return LBM_ERR_RANGE;
    }
    if (st & LBM_ST_OVERFLOW) {
        msg = "immersed boundary: correction patch overflow";
        return LBM_ERR_RANGE;
    }
    if (st & LBM_ST_SOLVER) {
        msg = "immersed boundary: D D^T not positive definite";
        return LBM_ERR_SOLVER;
    }
    if (st & LBM_ST_NONFINITE) {
        msg = "non-finite flow at the markers or force (the flow diverged)";
        return LBM_ERR_NONFINITE;
    }
    msg = "unknown device status";
    return LBM_ERR_CUDA;
}

namespace {

// Pinned host memory of a handle: what a call reads back goes there in one copy
// (a copy into pageable memory holds up the host for some 10 us; a step call
// made two). Blocks of destroyed handles are kept for the next ones, up to
// kHostBlocks of them.
constexpr size_t kHostBlock = 16384;
constexpr size_t kHostBlocks = 64;
std::mutex g_host_mu;
std::vector<void *> g_host_free;

void *host_block()
{
    {
        std::lock_guard<std::mutex> lock(g_host_mu);
        if (!g_host_free.empty()) {
            void *p = g_host_free.back();
            g_host_free.pop_back();
            return p;
        }
    }
    void *p = nullptr;
    if (cudaHostAlloc(&p, kHostBlock, cudaHostAllocPortable) == cudaSuccess) return p;
    cudaGetLastError();
    return nullptr;
}

void host_block_free(void *p)
{
    if (!p) return;
    {
        std::lock_guard<std::mutex> lock(g_host_mu);
        if (g_host_free.size() < kHostBlocks) {
            g_host_free.push_back(p);
            return;
        }
    }
    cudaFreeHost(p);
}

// rows that fit into the handle's block with the head
bool rows_fit(const lbm_handle *h, int rows)
{
    return sizeof(RunHead) + sizeof(double) * h->row_len * (size_t)rows <= kHostBlock;
}

int mass_result(lbm_handle *h, double dsum)
{
    const double m = (double)h->nx * (double)h->ny + dsum;   // sum_k w_k = 1 per node
    h->last_mass = m;
    h->last_mass_step = h->steps_done;
    if (!std::isfinite(m)) return set_err(h, LBM_ERR_NONFINITE, "mass check: non-finite populations (the flow diverged)");
    return LBM_OK;
}

int fetch(lbm_handle *h, cudaStream_t st, bool mass, int rows, double *dst)
{
    // the global mass check: the FP64 deviation sum of the current populations
    if (mass && launch_mass(h, h->fbuf[h->cur], st)) return cuda_err(h, cudaGetLastError(), "launch mass");
    const bool fit = dst && rows_fit(h, rows);
    const size_t bytes = sizeof(double) * h->row_len * (size_t)rows;
    CK(cudaMemcpyAsync(h->hblock, h->d_head, sizeof(RunHead) + (fit ? bytes : 0), cudaMemcpyDeviceToHost, st), "read status");
    if (dst && !fit) CK(cudaMemcpyAsync(dst, h->d_ring, bytes, cudaMemcpyDeviceToHost, st), "copy force rows");
    return LBM_OK;
}

int fetched(lbm_handle *h, bool mass, int rows, double *dst)
{
    const RunHead *head = (const RunHead *)h->hblock;
    if (dst && rows_fit(h, rows)) memcpy(dst, head + 1, sizeof(double) * h->row_len * (size_t)rows);
    if (const unsigned st = head->status) {
        CK(cudaMemsetAsync(h->d_status, 0, sizeof(unsigned), h->stream), "clear status");
        if (st & LBM_ST_TIMEOUT) CK(loop_reset(h), "reset step loop");
        std::string msg;
        const int code = status_error(st, msg);
        return set_err(h, code, msg.c_str());
    }
    return mass ? mass_result(h, head->mass) : LBM_OK;
}

// sums the event intervals of `count` step slots after the streams are idle:
// step time is the span from the first step's start to the last step's end
// (gaps between launches included); the lattice time is the sum of the
// lattice kernels' intervals; the IB time is measured on the stream it ran on
int collect_timing(lbm_handle *h, int count, bool split)
{
    if (count < 1) return LBM_OK;
    for (int s = 0; s < count && h->timing == LBM_TIMING_KERNELS; ++s) {
        float a = 0, b = 0, c = 0;
        CK(cudaEventElapsedTime(&a, h->ev[4 * s], h->ev[4 * s + 1]), "event time");
        CK(cudaEventElapsedTime(&b, h->ev[4 * s + 2], h->ev[4 * s + 3]), "event time");
        if (split) {
            CK(cudaEventElapsedTime(&c, h->ev_side[2 * s], h->ev_side[2 * s + 1]), "event time");
            h->t_kf += a + b;
            h->t_ib += c;
        } else {
            h->t_ib += a;
            h->t_kf += b;
        }
    }
    h->t_steps += count;
    float span = 0;
    CK(cudaEventElapsedTime(&span, h->ev[0], h->ev[4 * (count - 1) + 3]), "event time");
    h->t_step += span;
    return LBM_OK;
}

// The per-step sequence. Without a body, or with the split off: IB chain,
// then the fused lattice update, on the main stream. With the split: the IB
// flow chain runs on the side stream (after the previous step) and its force
// row and residual check on the check stream, while the main stream updates
// every node outside the step's correction tiles; the main stream's step
// ends once the side stream has updated the correction tiles.
int run_steps(lbm_handle *h, int nsteps, double *rows_out, int *done_out, bool fields_every)
{
    // the mass is checked at every copy of force rows of lbm_run (every
    // kRing steps and at the end of the call), and by lbm_step on every
    // kRing-th step
    auto mass_due = [&]() { return !fields_every || (h->n - 1) % kRing == 0; };
    if (!h->inited) return set_err(h, LBM_ERR_STATE, "step: lbm_init not called");
    for (int w = 0; w < h->nwing; ++w)
        if (!h->have_wing[w]) return set_err(h, LBM_ERR_STATE, "step: boundary of a wing not set");
    int rc = ensure_ib(h);
    if (rc) return rc;
    const bool split = h->overlap && h->nseg > 0 && h->env_w > 0 && h->env_h > 0;
    if (split) CK(cudaEventRecord(h->ev_inner, h->stream), "event");
    // Factorization of batch b (steps b*K .. b*K+K-1 that the motion table
    // reaches, into slot half b & 1). With the split it runs on the factor
    // stream once the half's previous user (the batch two back) is done;
    // otherwise in order on the main stream.
    const double dt_time = h->p.scale * h->p.uu;
    const int K = h->fbatch;
    // last step with time <= mend, plus one against rounding (factorizing a
    // step that is never run costs nothing but time)
    const int last_step = (int)std::floor((h->mend + 1.0e-12) / dt_time) + 2;
    auto factor_batch = [&](int b) -> int {
        const int half = b & 1;
        const int s0 = std::max(1, b * K), s1 = std::min(b * K + K - 1, last_step);
        h->batch_in_half[half] = b;
        if (h->nseg == 0 || s1 < s0) return LBM_OK;
        cudaStream_t st = split ? h->fstream : h->stream;
        // the half's previous users: the flow chains and checks of its steps
        // (ev_free) and the lattice kernels of those steps on the main stream,
        // which read the slots' patch rectangles and tile counts (ev_inner:
        // the main stream's last completed step)
        if (split) {
            CK(cudaStreamWaitEvent(h->fstream, h->ev_free[half], 0), "wait");
            CK(cudaStreamWaitEvent(h->fstream, h->ev_inner, 0), "wait");
        }
        if (launch_factor(h, s0, s1 - s0 + 1, st)) return cuda_err(h, cudaGetLastError(), "launch factor");
        if (h->pairs) {
            if (launch_near_cells(h, s0, s1 - s0 + 1, st)) return cuda_err(h, cudaGetLastError(), "launch near cells");
            h->near_in_half[half] = b;
        }
        if (split) CK(cudaEventRecord(h->ev_batch[half], h->fstream), "event");
        return LBM_OK;
    };
    // The near cells of batch b where its half was factorized without them, by
    // an lbm_batch (whose run has ended: nothing of its is queued). They
    // replace those of the batch two back, which the factor stream waits for
    // as factor_batch does.
    auto near_batch = [&](int b) -> int {
        const int half = b & 1;
        const int s0 = std::max(1, b * K), s1 = std::min(b * K + K - 1, last_step);
        CK(cudaStreamWaitEvent(h->fstream, h->ev_free[half], 0), "wait");
        CK(cudaStreamWaitEvent(h->fstream, h->ev_inner, 0), "wait");
        if (launch_near_cells(h, s0, s1 - s0 + 1, h->fstream)) return cuda_err(h, cudaGetLastError(), "launch near cells");
        h->near_in_half[half] = b;
        CK(cudaEventRecord(h->ev_batch[half], h->fstream), "event");
        return LBM_OK;
    };
    // The next batch's factorization runs beside this batch's steps; a call that
    // ends in the first half of a batch leaves it to a later one.
    auto factor_next = [&](int b, int s) -> int {
        if ((b + 1) * K > last_step || h->batch_in_half[(b + 1) & 1] == b + 1 || h->n % K + (nsteps - s) <= K / 2) return LBM_OK;
        return factor_batch(b + 1);
    };
    int done = 0, pending = 0;
    // step n has a successor in the motion
    auto goes_on = [&](int n) { return (double)n * dt_time <= h->mend + 1.0e-12; };
    // a small lattice's steps run as step_loop launches; per-kernel timing
    // needs the kernels one by one
    const bool loop = split && h->timing != LBM_TIMING_KERNELS && loop_fits(h);
    const bool pairs = split && !loop && h->pairs && h->timing != LBM_TIMING_KERNELS;
    bool joined = loop;   // nothing queued on the side and check streams since the last flush
    // force rows, mass check, status and timing of the steps since the last flush
    auto flush = [&]() -> int {
        if (split && !joined) {   // force rows and residual checks run on the check stream after the update
            CK(cudaEventRecord(h->ev_ib, h->side), "event");
            CK(cudaStreamWaitEvent(h->stream, h->ev_ib, 0), "wait");
            CK(cudaEventRecord(h->ev_cjoin, h->cstream), "event");
            CK(cudaStreamWaitEvent(h->stream, h->ev_cjoin, 0), "wait");
            joined = loop;
        }
        // the span ends with the chunk's last step; the row copy and the
        // mass check after it are per-call work, not per-step work
        if (h->timing == LBM_TIMING_SPAN) CK(cudaEventRecord(h->ev[4 * (pending - 1) + 3], h->stream), "event");
        const bool mass = mass_due();
        double *dst = rows_out ? rows_out + (size_t)(done - pending) * h->row_len : nullptr;
        int st = fetch(h, h->stream, mass, pending, dst);
        if (st) return st;
        CK(cudaStreamSynchronize(h->stream), "step sync");
        if ((st = fetched(h, mass, pending, dst))) return st;
        if (h->timing && (st = collect_timing(h, pending, split))) return st;
        pending = 0;
        return LBM_OK;
    };
    rc = LBM_OK;
    for (int s = 0; s < nsteps; ++s) {
        const double time = (double)(h->n - 1) * dt_time;   // main.f90:352
        if (time > h->mend + 1.0e-12) { rc = LBM_DONE; break; }
        if (loop) {
            // as many steps as the slot half, the force ring, the call and the
            // motion hold, in one launch
            const int b = h->n / K, half = b & 1;
            int m = 1;
            while (m < nsteps - s && (h->n + m) / K == b && pending + m < h->ring_cap && goes_on(h->n + m - 1)) ++m;
            if (h->batch_in_half[half] != b && (rc = factor_batch(b))) return rc;
            // the next batch's factorization, beside this launch (it waits for
            // the previous one, not for this one)
            if ((rc = factor_next(b, s))) return rc;
            void *fields[LBM_NSLOT_MAX] = {};
            for (int t = 0; t < m; ++t)
                if (fields_every || s + t >= nsteps - 2) {
                    const int fs = h->fields_slot ^ 1;
                    fields[t] = h->d_fields[fs];
                    h->fields_slot = fs;
                    h->fields_step[fs] = h->n + t;
                }
            if (h->timing == LBM_TIMING_SPAN && pending == 0) CK(cudaEventRecord(h->ev[0], h->stream), "event");
            CK(cudaStreamWaitEvent(h->stream, h->ev_batch[half], 0), "wait");
            if (launch_loop(h, m, fields, h->stream)) return cuda_err(h, cudaGetLastError(), "launch step loop");
            CK(cudaEventRecord(h->ev_inner, h->stream), "event");
            // force rows and residual checks beside the next launch; those of
            // a call that is one launch have nothing to run beside
            cudaStream_t cs = joined && s + m == nsteps ? h->stream : h->cstream;
            if (cs != h->stream) {
                CK(cudaStreamWaitEvent(cs, h->ev_inner, 0), "wait");
                joined = false;
            }
            if (launch_check_steps(h, h->n, m, pending, s + m == nsteps || !goes_on(h->n + m - 1), cs))
                return cuda_err(h, cudaGetLastError(), "launch check");
            CK(cudaEventRecord(h->ev_free[half], cs), "event");
            if (m & 1) h->cur ^= 1;
            h->n += m;
            h->steps_done += m;
            done += m;
            pending += m;
            s += m - 1;
            if (pending == h->ring_cap || s == nsteps - 1)
                if ((rc = flush())) return rc;
            continue;
        }
        // two steps at once: an even one and the next, neither keeping fields
        if (pairs && h->n % 2 == 0 && s + 1 < nsteps - 2 && pending + 1 < h->ring_cap && goes_on(h->n)) {
            const int slot = pending, b = h->n / K, half = b & 1;
            const void *fin = h->fbuf[h->cur];
            void *fout = h->fbuf[h->cur ^ 1];
            if (h->batch_in_half[half] != b && (rc = factor_batch(b))) return rc;
            if (h->near_in_half[half] != b && (rc = near_batch(b))) return rc;
            if (h->timing == LBM_TIMING_SPAN && slot == 0) CK(cudaEventRecord(h->ev[0], h->stream), "event");
            for (cudaStream_t st : {h->side, h->nstream}) {
                CK(cudaStreamWaitEvent(st, h->ev_inner, 0), "wait");
                CK(cudaStreamWaitEvent(st, h->ev_batch[half], 0), "wait");
            }
            cudaEvent_t ei = h->after_interp ? h->ev_interp : nullptr;
            const void *src = fin;
            for (int t = 0; t < 2; ++t) {
                void *dst = t ? fout : h->fmid;
                const int q = h->n % h->nslots;
                h->pinfo_slot = q;
                // the flow chain and the correction tiles; beside them the
                // other nodes near the bodies (the second step's after the
                // first step's tiles)
                if (t) {
                    CK(cudaStreamWaitEvent(h->side, h->ev_near[0], 0), "wait");
                    CK(cudaStreamWaitEvent(h->nstream, h->ev_ib, 0), "wait");
                }
                if (launch_near(h, src, dst, h->n - t, t, h->nstream)) return cuda_err(h, cudaGetLastError(), "launch near");
                CK(cudaEventRecord(h->ev_near[t], h->nstream), "event");
                if (launch_flow(h, src, dst, nullptr, h->n, slot + t, q, h->side, t ? nullptr : ei)) return cuda_err(h, cudaGetLastError(), "launch ib");
                CK(cudaEventRecord(h->ev_ib, h->side), "event");
                CK(cudaStreamWaitEvent(h->cstream, h->ev_ib, 0), "wait");
                if (launch_check(h, h->n, slot + t, check_due(h->n) || !goes_on(h->n), h->cstream)) return cuda_err(h, cudaGetLastError(), "launch check");
                if (t == 0) {
                    if ((rc = factor_next(b, s))) return rc;
                    CK(cudaStreamWaitEvent(h->stream, h->ev_batch[half], 0), "wait");
                    if (ei) CK(cudaStreamWaitEvent(h->stream, ei, 0), "wait");   // the solve starts first
                    if (launch_pair(h, fin, fout, h->stream)) return cuda_err(h, cudaGetLastError(), "launch pair");
                    h->count(2, 1);   // the lattice, for both steps
                }
                src = dst;
                h->n++;
            }
            CK(cudaEventRecord(h->ev_free[half], h->cstream), "event");
            CK(cudaStreamWaitEvent(h->stream, h->ev_ib, 0), "wait");
            CK(cudaStreamWaitEvent(h->stream, h->ev_near[1], 0), "wait");
            CK(cudaEventRecord(h->ev_inner, h->stream), "event");   // both steps are complete
            h->cur ^= 1;
            h->steps_done += 2;
            done += 2;
            pending += 2;
            s += 1;
            if (pending == h->ring_cap || s == nsteps - 1)
                if ((rc = flush())) return rc;
            continue;
        }
        const int slot = pending, b = h->n / K, half = b & 1, q = h->n % h->nslots;
        h->pinfo_slot = q;
        const void *fin = h->fbuf[h->cur];
        void *fout = h->fbuf[h->cur ^ 1];
        void *fields = nullptr;
        const bool want = fields_every || s >= nsteps - 2;
        if (want) {
            const int fs = h->fields_slot ^ 1;
            fields = h->d_fields[fs];
            h->fields_slot = fs;
            h->fields_step[fs] = h->n;
        }
        // per-step events (LBM_TIMING_KERNELS); with LBM_TIMING_SPAN only the
        // first step's start and the last step's end of each chunk of steps
        cudaEvent_t *e = h->timing == LBM_TIMING_KERNELS ? &h->ev[4 * slot] : nullptr;
        if (h->timing == LBM_TIMING_SPAN && slot == 0) CK(cudaEventRecord(h->ev[0], h->stream), "event");
        // the solve-residual check: on every kCheckEvery-th step and on the
        // last step of the call or of the motion
        const bool check_res = check_due(h->n) || s == nsteps - 1 || !goes_on(h->n);
        if (split) {
            // side stream: the immersed-boundary chain and the correction
            // tiles; main stream: every other node, concurrently
            if (h->batch_in_half[half] != b && (rc = factor_batch(b))) return rc;
            CK(cudaStreamWaitEvent(h->side, h->ev_inner, 0), "wait");
            CK(cudaStreamWaitEvent(h->side, h->ev_batch[half], 0), "wait");
            if (e) CK(cudaEventRecord(h->ev_side[2 * slot], h->side), "event");
            cudaEvent_t ei = h->after_interp ? h->ev_interp : nullptr;
            if (launch_flow(h, fin, fout, fields, h->n, slot, q, h->side, ei)) return cuda_err(h, cudaGetLastError(), "launch ib");
            if (e) CK(cudaEventRecord(h->ev_side[2 * slot + 1], h->side), "event");
            CK(cudaEventRecord(h->ev_ib, h->side), "event");
            // the force row and the residual check on their own stream; the
            // slot half is free for the next factorization after them
            CK(cudaStreamWaitEvent(h->cstream, h->ev_ib, 0), "wait");
            if (launch_check(h, h->n, slot, check_res, h->cstream)) return cuda_err(h, cudaGetLastError(), "launch check");
            CK(cudaEventRecord(h->ev_free[half], h->cstream), "event");
            if ((rc = factor_next(b, s))) return rc;
            CK(cudaStreamWaitEvent(h->stream, h->ev_batch[half], 0), "wait");   // the step's correction tiles
            if (ei) CK(cudaStreamWaitEvent(h->stream, ei, 0), "wait");   // the solve starts first
            if (e) CK(cudaEventRecord(e[0], h->stream), "event");
            if (launch_kf(h, fin, fout, fields, KF_OUTER)) return cuda_err(h, cudaGetLastError(), "launch kf");
            if (e) CK(cudaEventRecord(e[1], h->stream), "event");
            CK(cudaStreamWaitEvent(h->stream, h->ev_ib, 0), "wait");
            if (e) {
                CK(cudaEventRecord(e[2], h->stream), "event");
                CK(cudaEventRecord(e[3], h->stream), "event");
            }
            CK(cudaEventRecord(h->ev_inner, h->stream), "event");   // the step is complete
        } else {
            if (e) CK(cudaEventRecord(e[0], h->stream), "event");
            if (h->batch_in_half[half] != b && (rc = factor_batch(b))) return rc;
            if (launch_flow(h, fin, fout, fields, h->n, slot, q, h->stream)) return cuda_err(h, cudaGetLastError(), "launch ib");
            if (launch_check(h, h->n, slot, check_res, h->stream)) return cuda_err(h, cudaGetLastError(), "launch check");
            if (e) {
                CK(cudaEventRecord(e[1], h->stream), "event");
                CK(cudaEventRecord(e[2], h->stream), "event");
            }
            if (launch_kf(h, fin, fout, fields, h->nseg > 0 ? KF_OUTER : KF_ALL)) return cuda_err(h, cudaGetLastError(), "launch kf");
            if (e) CK(cudaEventRecord(e[3], h->stream), "event");
        }
        h->cur ^= 1;
        h->n++;
        h->steps_done++;
        done++;
        pending++;
        if (pending == h->ring_cap || s == nsteps - 1) {
            const int st = flush();
            if (st) return st;
        }
    }
    if (pending) {
        const int st = flush();
        if (st) return st;
    }
    if (done_out) *done_out = done;
    return rc;
}

}  // namespace

// an empty kernel, compiled like every other kernel of the library: its
// attributes tell which architecture the library's device code is for
__global__ void arch_probe() {}

// The errors of the steps discarded go with them: the next user of a slot
// would report what no step of its own has seen.
void forget_batches(lbm_handle *h)
{
    for (int q = 0; q < 2; ++q) h->batch_in_half[q] = h->near_in_half[q] = h->fgroup[q] = -1;
    if (h->d_fstatus) cudaMemsetAsync(h->d_fstatus, 0, sizeof(unsigned) * h->nslots, h->stream);
}

// for lbm_batch.cu
int handle_prepare_ib(lbm_handle *h) { return ensure_ib(h); }
int handle_fetch(lbm_handle *h, cudaStream_t st, bool mass, int rows, double *dst) { return fetch(h, st, mass, rows, dst); }
int handle_fetched(lbm_handle *h, bool mass, int rows, double *dst) { return fetched(h, mass, rows, dst); }
int handle_error(lbm_handle *h, int code, const char *msg) { return set_err(h, code, msg); }

// boundary reference values from the edge f0 (FP64, full f; left column,
// right column, bottom row, top row, 9 per node): the moments
// physical_variables takes on the edge columns (solution.f90:516-520) and the
// corner-column f0 populations the top/bottom extrapolation reads
// (boundary_condition.f90:705, 832)
int handle_set_edges(lbm_handle *h, const double *ef)
{
    const int nx = h->nx, ny = h->ny;
    std::vector<double> ec(6 * (size_t)ny + 36);
    for (int side = 0; side < 2; ++side) {
        for (int j = 0; j < ny; ++j) {
            const double *f = ef + 9 * ((size_t)side * ny + j);
            double temprho = 0.0, tempu = 0.0, tempv = 0.0;
            for (int k = 0; k < 9; ++k) {
                temprho = temprho + f[k];
                tempu = tempu + (double)kEx[k] * f[k];
                tempv = tempv + (double)kEy[k] * f[k];
            }
            double *o = ec.data() + (size_t)side * 3 * ny + 3 * (size_t)j;
            o[0] = temprho - 1.0;
            o[1] = tempu / temprho;
            o[2] = tempv / temprho;
        }
    }
    // (1,2), (1,Ny-1), (Nx,2), (Nx,Ny-1) as deviations from the weights
    const int cside[4] = {0, 0, 1, 1}, cj[4] = {1, ny - 2, 1, ny - 2};
    for (int c = 0; c < 4; ++c) {
        const double *f = ef + 9 * ((size_t)cside[c] * ny + cj[c]);
        for (int k = 0; k < 9; ++k) ec[6 * (size_t)ny + 9 * c + k] = f[k] - kWref[k];
    }
    if (compute_size(h->prec) == sizeof(double)) {
        CK(cudaMemcpyAsync(h->edge_c, ec.data(), sizeof(double) * ec.size(), cudaMemcpyHostToDevice, h->stream), "copy edge");
        CK(cudaStreamSynchronize(h->stream), "sync edge");
    } else {
        std::vector<float> ecf(ec.begin(), ec.end());
        CK(cudaMemcpyAsync(h->edge_c, ecf.data(), sizeof(float) * ecf.size(), cudaMemcpyHostToDevice, h->stream), "copy edge");
        CK(cudaStreamSynchronize(h->stream), "sync edge");
    }
    h->edge_f0.assign(ef, ef + 9 * (2 * (size_t)ny + 2 * (size_t)nx));
    return LBM_OK;
}

// readflowfield (solution.f90:1709-1839) on the device: f is packed into the
// storage precision, the field slot gets u and v with density 1 (init's
// rho0; the file has no density), the boundary values come from the edge f0,
// and the step counter continues after `cycle` (main.f90:321-323: n = cycle1
// + 1). The factorization slots are filled again for the restored step.
int handle_restore(lbm_handle *h, const double *f, const double *u, const double *v, const double *edge_f0, int cycle)
{
    quiesce(h);
    const size_t nn = (size_t)h->nx * h->ny;
    if (!h->d_stage) CK(dmalloc(h, &h->d_stage, sizeof(double) * nn * 9), "alloc stage");
    CK(cudaMemcpyAsync(h->d_stage, f, sizeof(double) * nn * 9, cudaMemcpyHostToDevice, h->stream), "copy f");
    if (launch_pack(h, h->d_stage, h->fbuf[0])) return cuda_err(h, cudaGetLastError(), "pack");
    CK(cudaStreamSynchronize(h->stream), "sync f");
    free_devp(h->d_stage);
    h->cur = 0;
    if (compute_size(h->prec) == sizeof(double)) {
        std::vector<double> fl(3 * nn);
        for (size_t q = 0; q < nn; ++q) {
            fl[q] = 1.0;
            fl[nn + q] = u[q];
            fl[2 * nn + q] = v[q];
        }
        CK(cudaMemcpyAsync(h->d_fields[0], fl.data(), sizeof(double) * fl.size(), cudaMemcpyHostToDevice, h->stream),
           "copy fields");
        CK(cudaStreamSynchronize(h->stream), "sync fields");
    } else {
        std::vector<float> fl(3 * nn);
        for (size_t q = 0; q < nn; ++q) {
            fl[q] = 1.0f;
            fl[nn + q] = (float)u[q];
            fl[2 * nn + q] = (float)v[q];
        }
        CK(cudaMemcpyAsync(h->d_fields[0], fl.data(), sizeof(float) * fl.size(), cudaMemcpyHostToDevice, h->stream),
           "copy fields");
        CK(cudaStreamSynchronize(h->stream), "sync fields");
    }
    const int rc = handle_set_edges(h, edge_f0);
    if (rc) return rc;
    CK(cudaMemsetAsync(h->d_status, 0, sizeof(unsigned), h->stream), "clear status");
    CK(cudaMemsetAsync(h->d_pinfo, 0, LBM_NSLOT_MAX * sizeof(PatchInfo), h->stream), "clear pinfo");
    CK(cudaStreamSynchronize(h->stream), "sync restore");
    h->n = cycle + 1;
    h->steps_done = cycle;
    h->fields_slot = 0;
    h->fields_step[0] = cycle;
    h->fields_step[1] = -1;
    forget_batches(h);
    return LBM_OK;
}

extern "C" {

int lbm_default_params(lbm_params *p)
{
    if (!p) return LBM_ERR_ARG;
    memset(p, 0, sizeof *p);
    p->nx = 4001;                 // nint(40/0.01)+1 (ini_mesh.f90:22)
    p->ny = 2001;                 // nint(20/0.01)+1 (ini_mesh.f90:23)
    p->wing_count = 2;            // main.f90:18
    p->points_per_wing = 205;     // main.f90:21
    p->delta_kernel = LBM_DELTA_SMOOTH;   // boundary_condition.f90:1530
    p->precision = LBM_PREC_FP32;
    p->scale = 0.01;              // mesh_max_scale (main.f90:32)
    p->ox = -20.0;                // -0.5*width (ini_mesh.f90:36)
    p->oy = -10.0;
    p->uu = 0.01;                 // main.f90:12
    p->re = 500.0;                // main.f90:84
    const double s[9] = {0.0, 1.1, 1.05, 0.0, 1.2, 0.0, 1.2, 0.0, 0.0};   // ini_mesh.f90:59-67
    memcpy(p->s, s, sizeof s);
    p->mesh_max_scale = 0.01;
    return LBM_OK;
}

int lbm_create(const lbm_params *p, lbm_t **out)
{
    if (!p || !out) return LBM_ERR_ARG;
    *out = nullptr;
    if (p->nx < 16 || p->ny < 16 || p->wing_count < 0 || p->wing_count > LBM_MAXW ||
        (p->wing_count > 0 && p->points_per_wing < 3) || !(p->scale > 0) || !(p->uu > 0) || !(p->re > 0) ||
        p->precision < 0 || p->precision > 3 || p->delta_kernel < 0 || p->delta_kernel > 1 || (p->flags & ~LBM_FLAG_DENSE_SOLVE) != 0 ||
        (long long)p->wing_count * (p->points_per_wing - 1) > ib_max_markers())
        return LBM_ERR_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1) return LBM_ERR_CUDA;
    lbm_handle *h = new lbm_handle();
    h->p = *p;
    cudaGetDevice(&h->dev);
    h->nx = p->nx;
    h->ny = p->ny;
    h->pitch = (p->nx + 63) / 64 * 64;
    h->plane = (long long)h->pitch * p->ny;
    h->nwing = p->wing_count;
    h->ppw = h->nwing > 0 ? p->points_per_wing : 0;
    h->spw = h->ppw > 0 ? h->ppw - 1 : 0;
    h->npts = h->nwing * h->ppw;
    h->nseg = h->nwing * h->spw;
    h->niu = p->uu * (1.0 / p->scale) / p->re;   // ini_mesh.f90:30
    h->tau = 3.0 * h->niu + 0.5;                  // ini_mesh.f90:31
    for (int k = 0; k < 9; ++k) h->s[k] = p->s[k];
    if (p->s[7] <= 0) h->s[7] = 1.0 / h->tau;
    if (p->s[8] <= 0) h->s[8] = 1.0 / h->tau;
    h->prec = p->precision;
    h->elem = storage_size(h->prec);
    // nodes per thread of the lattice kernel; LBM_KF_VEC (1, 2 or 4) overrides
    // the default for tuning
    h->kf_vec = 1;
    if (const char *ev = getenv("LBM_KF_VEC")) {
        const int v = atoi(ev);
        if (v == 1 || v == 2 || v == 4) h->kf_vec = v;
    }
    if (const char *ev = getenv("LBM_KF_TMA")) h->kf_tma = atoi(ev) != 0;

    if (const char *ev = getenv("LBM_KF_ROWS")) {
        const int v = atoi(ev);
        if (v >= 1 && v <= 4096) h->kf_rows = v;
    }
    h->hx0.assign(std::max(1, h->npts), 0.0);
    h->hy0.assign(std::max(1, h->npts), 0.0);
    h->harc.assign(std::max(1, h->nseg), 0.0);
    h->have_wing.assign(LBM_MAXW, 0);
    h->row_len = 1 + 3 * h->nwing + 3 + 9 * h->nwing;
    h->ring_cap = kRing;
    auto fail = [&](cudaError_t e, const char *w) {
        lbm_destroy(h);
        (void)e; (void)w;
        return LBM_ERR_CUDA;
    };
    cudaError_t e;
    if ((e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking)) != cudaSuccess) return fail(e, "stream");
    // the immersed-boundary flow chain is on the step's critical path: its
    // stream has the highest priority, so that its CTAs are placed before
    // queued lattice CTAs as SMs free up
    int prio_low = 0, prio_high = 0;
    if ((e = cudaDeviceGetStreamPriorityRange(&prio_low, &prio_high)) != cudaSuccess) return fail(e, "priorities");
    if ((e = cudaStreamCreateWithPriority(&h->side, cudaStreamNonBlocking, prio_high)) != cudaSuccess)
        return fail(e, "side stream");
    if ((e = cudaEventCreateWithFlags(&h->ev_ib, cudaEventDisableTiming)) != cudaSuccess) return fail(e, "event");
    if ((e = cudaEventCreateWithFlags(&h->ev_inner, cudaEventDisableTiming)) != cudaSuccess) return fail(e, "event");
    if ((e = cudaEventCreateWithFlags(&h->ev_interp, cudaEventDisableTiming)) != cudaSuccess) return fail(e, "event");
    if (const char *ev = getenv("LBM_AFTER_INTERP")) h->after_interp = atoi(ev) != 0;
    if ((e = cudaStreamCreateWithFlags(&h->fstream, cudaStreamNonBlocking)) != cudaSuccess) return fail(e, "factor stream");
    if ((e = cudaStreamCreateWithPriority(&h->cstream, cudaStreamNonBlocking, prio_high)) != cudaSuccess)
        return fail(e, "check stream");
    if ((e = cudaEventCreateWithFlags(&h->ev_cjoin, cudaEventDisableTiming)) != cudaSuccess) return fail(e, "event");
    for (int q = 0; q < 2; ++q) {
        if ((e = cudaEventCreateWithFlags(&h->ev_batch[q], cudaEventDisableTiming)) != cudaSuccess) return fail(e, "event");
        if ((e = cudaEventCreateWithFlags(&h->ev_free[q], cudaEventDisableTiming)) != cudaSuccess) return fail(e, "event");
    }
    if (const char *ov = getenv("LBM_OVERLAP")) h->overlap = atoi(ov) != 0;
    if (const char *fb = getenv("LBM_IB_BATCH")) {
        const int v = atoi(fb);
        if (v >= 1 && 2 * v <= LBM_NSLOT_MAX) h->fbatch = v;
    }
    h->nslots = 2 * h->fbatch;
    {
        // a CTA of the step loop fills an SM; kLoopSpare SMs stay free for the
        // factorization of the next steps, which runs beside it
        int sms = 0, coop = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->dev);
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, h->dev);
        h->loop_ctas = coop && h->overlap && h->kf_tma ? std::max(0, sms - kLoopSpare) : 0;
    }
    // population buffers carry LBM_FPAD elements of padding before and after
    // the 9 planes, so the bulk row copies of the lattice kernel (which read a
    // 16-byte halo left and right of every row segment) stay in bounds
    const size_t fbytes = h->elem * (9 * (size_t)h->plane + 2 * LBM_FPAD);
    for (int b = 0; b < 2; ++b) {
        if ((e = dmalloc(h, &h->falloc[b], fbytes)) != cudaSuccess) return fail(e, "alloc f");
        h->fbuf[b] = (char *)h->falloc[b] + h->elem * LBM_FPAD;
    }
    const size_t cs = compute_size(h->prec);
    const size_t nn = (size_t)h->nx * h->ny;
    for (int b = 0; b < 2; ++b)
        if ((e = dmalloc(h, &h->d_fields[b], 3 * cs * nn)) != cudaSuccess) return fail(e, "alloc fields");
    if ((e = dmalloc(h, &h->edge_c, cs * (6 * (size_t)h->ny + 36))) != cudaSuccess) return fail(e, "alloc edge");
    if ((e = dmalloc(h, &h->d_pinfo, LBM_NSLOT_MAX * sizeof(PatchInfo))) != cudaSuccess) return fail(e, "alloc pinfo");
    if ((e = dmalloc(h, &h->d_red, sizeof(double) * 2 * 296)) != cudaSuccess) return fail(e, "alloc red");
    if ((e = dmalloc(h, &h->d_mass, sizeof(double) * mass_slots())) != cudaSuccess) return fail(e, "alloc mass");
    if ((e = dmalloc(h, &h->d_mcount, sizeof(unsigned))) != cudaSuccess) return fail(e, "alloc mass counter");

    // solve residual and half-bandwidth, per slot
    if ((e = dmalloc(h, &h->d_solve_res, LBM_NSLOT_MAX * 2 * sizeof(double))) != cudaSuccess) return fail(e, "alloc res");
    if ((e = dmalloc(h, &h->d_sync, sizeof(unsigned) * loop_sync_words())) != cudaSuccess) return fail(e, "alloc sync");
    if ((e = dmalloc(h, &h->d_head, sizeof(RunHead) + sizeof(double) * h->row_len * (size_t)h->ring_cap)) != cudaSuccess)
        return fail(e, "alloc ring");
    h->d_status = &h->d_head->status;
    h->d_ring = (double *)(h->d_head + 1);
    if (!(h->hblock = host_block())) return fail(cudaErrorMemoryAllocation, "alloc host block");
    if (h->npts > 0) {
        if ((e = dmalloc(h, &h->d_xb0, sizeof(double) * h->npts)) != cudaSuccess) return fail(e, "alloc xb0");
        if ((e = dmalloc(h, &h->d_yb0, sizeof(double) * h->npts)) != cudaSuccess) return fail(e, "alloc yb0");
        if ((e = dmalloc(h, &h->d_arc, sizeof(double) * h->nseg)) != cudaSuccess) return fail(e, "alloc arc");
    }
    // the zero-fills queued on the handle's stream are done (later calls
    // order their work after them on the same stream in any case)
    if ((e = cudaStreamSynchronize(h->stream)) != cudaSuccess) return fail(e, "sync");
    *out = h;
    return LBM_OK;
}

int lbm_destroy(lbm_t *h)
{
    if (!h) return LBM_ERR_ARG;
    // no queued work of the handle may still use what is freed below
    if (h->fstream) cudaStreamSynchronize(h->fstream);
    if (h->side) cudaStreamSynchronize(h->side);
    if (h->cstream) cudaStreamSynchronize(h->cstream);
    if (h->nstream) cudaStreamSynchronize(h->nstream);
    if (h->stream) cudaStreamSynchronize(h->stream);
    for (int b = 0; b < 2; ++b) { free_dev(h->falloc[b]); h->fbuf[b] = nullptr; free_dev(h->d_fields[b]); }
    free_dev(h->edge_c);
    free_devp(h->d_xb0); free_devp(h->d_yb0); free_devp(h->d_arc); free_devp(h->d_mstep);
    free_ib(h);
    free_devp(h->d_pinfo); 
    free_devp(h->d_head); free_devp(h->d_solve_res);
    host_block_free(h->hblock);
    free_devp(h->d_red);
    free_devp(h->d_mass); free_devp(h->d_mcount); free_devp(h->d_sync);

    free_devp(h->d_stage);
    if (h->side) cudaStreamSynchronize(h->side);
    if (h->cstream) cudaStreamSynchronize(h->cstream);
    if (h->nstream) cudaStreamSynchronize(h->nstream);
    if (h->fstream) cudaStreamSynchronize(h->fstream);
    // the frees above went to the pool on the main stream: once they have
    // completed, an allocation on any other stream may reuse the memory (one
    // made before the driver has seen them complete maps new memory instead)
    if (h->stream) cudaStreamSynchronize(h->stream);
    for (auto &e : h->ev) cudaEventDestroy(e);
    for (auto &e : h->ev_side) cudaEventDestroy(e);
    if (h->ev_ib) cudaEventDestroy(h->ev_ib);
    if (h->ev_inner) cudaEventDestroy(h->ev_inner);
    if (h->ev_interp) cudaEventDestroy(h->ev_interp);
    for (int q = 0; q < 2; ++q) {
        if (h->ev_near[q]) cudaEventDestroy(h->ev_near[q]);
        if (h->ev_batch[q]) cudaEventDestroy(h->ev_batch[q]);
        if (h->ev_free[q]) cudaEventDestroy(h->ev_free[q]);
    }
    if (h->ev_cjoin) cudaEventDestroy(h->ev_cjoin);
    if (h->nstream) cudaStreamDestroy(h->nstream);
    if (h->cstream) cudaStreamDestroy(h->cstream);
    if (h->fstream) cudaStreamDestroy(h->fstream);
    if (h->side) cudaStreamDestroy(h->side);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
    return LBM_OK;
}

int lbm_set_boundary(lbm_t *h, int wing, const double *x, const double *y, int npts)
{
    if (!h) return LBM_ERR_ARG;
    quiesce(h);   // queued work may still read what is rewritten below
    if (wing < 1 || wing > h->nwing || !x || !y || npts != h->ppw)
        return set_err(h, LBM_ERR_ARG, "set_boundary: bad wing index or point count");
    const int ps = (wing - 1) * h->ppw, ss = (wing - 1) * h->spw;
    for (int i = 0; i < npts; ++i) {
        if (!std::isfinite(x[i]) || !std::isfinite(y[i])) return set_err(h, LBM_ERR_ARG, "set_boundary: non-finite point");
        h->hx0[ps + i] = x[i];
        h->hy0[ps + i] = y[i];
    }
    for (int i0 = 0; i0 < h->spw; ++i0) {                 // airfoil.f90:235-238
        const double dx = h->hx0[ps + i0 + 1] - h->hx0[ps + i0];
        const double dy = h->hy0[ps + i0 + 1] - h->hy0[ps + i0];
        h->harc[ss + i0] = sqrt(dx * dx + dy * dy) / h->p.scale;
    }
    for (int i = 0; i < npts; ++i) {                      // airfoil.f90:240-241
        h->hx0[ps + i] = h->hx0[ps + i] + (h->p.xc - h->p.xp);
        h->hy0[ps + i] = h->hy0[ps + i] + (h->p.yc - h->p.yp);
    }
    CK(cudaMemcpyAsync(h->d_xb0 + ps, h->hx0.data() + ps, sizeof(double) * npts, cudaMemcpyHostToDevice, h->stream), "copy xb0");
    CK(cudaMemcpyAsync(h->d_yb0 + ps, h->hy0.data() + ps, sizeof(double) * npts, cudaMemcpyHostToDevice, h->stream), "copy yb0");
    CK(cudaMemcpyAsync(h->d_arc + ss, h->harc.data() + ss, sizeof(double) * h->spw, cudaMemcpyHostToDevice, h->stream), "copy arc");
    CK(cudaStreamSynchronize(h->stream), "sync boundary");
    h->have_wing[wing - 1] = 1;
    free_ib(h);
    return LBM_OK;
}

int lbm_set_motion_table(lbm_t *h, const double *table, int rows, int cols)
{
    if (!h) return LBM_ERR_ARG;
    quiesce(h);   // queued work may still read what is rewritten below
    if (!table) return set_err(h, LBM_ERR_ARG, "motion table: null");
    if (cols != 1 + 9 * h->nwing) return set_err(h, LBM_ERR_IO, "motion table: column count must be 1+9*wing_count");
    if (rows < 1) return set_err(h, LBM_ERR_IO, "motion table: empty");          // mode.f90:101-104
    for (int r = 1; r < rows; ++r)                                                 // mode.f90:130-135
        if (table[r] < table[r - 1]) return set_err(h, LBM_ERR_IO, "motion table: time column must be non-decreasing");
    for (size_t q = 0; q < (size_t)rows * cols; ++q)
        if (!std::isfinite(table[q])) return set_err(h, LBM_ERR_IO, "motion table: non-finite value");
    h->mtab.assign(table, table + (size_t)rows * cols);
    h->mrows = rows;
    h->mcols = cols;
    h->mend = table[rows - 1];                                                     // mode.f90:127
    h->mdt = h->p.scale * h->p.uu;                                                 // main.f90:255
    h->msteps = (int)((h->mend + 1.0e-12) / h->mdt) + 1;                           // mode.f90:258
    h->mstep_host.assign((size_t)h->msteps * cols, 0.0);
    int idx = 0;
    std::vector<double> row(cols);
    for (int i = 1; i <= h->msteps; ++i) {                                         // mode.f90:263-268
        lookup_row(h->mtab, rows, cols, (double)(i - 1) * h->mdt, idx, row.data());
        std::copy(row.begin(), row.end(), h->mstep_host.begin() + (size_t)(i - 1) * cols);
    }
    free_devp(h->d_mstep);
    CK(dmalloc(h, &h->d_mstep, sizeof(double) * h->mstep_host.size()), "alloc step table");
    CK(cudaMemcpyAsync(h->d_mstep, h->mstep_host.data(), sizeof(double) * h->mstep_host.size(),
                       cudaMemcpyHostToDevice, h->stream), "copy step table");
    CK(cudaStreamSynchronize(h->stream), "sync motion");
    free_ib(h);
    return LBM_OK;
}

int lbm_init(lbm_t *h, const double *du, const double *dv)
{
    if (!h) return LBM_ERR_ARG;
    if (h->mstep_host.empty()) return set_err(h, LBM_ERR_STATE, "init: motion table not loaded (mode.f90:275-276)");
    quiesce(h);   // queued work may still read what is rewritten below
    const int nx = h->nx, ny = h->ny;
    const size_t nn = (size_t)nx * ny;
    // initial f = feq(rho=1, u=UU(+du), v=0(+dv)) with single-precision weights
    // (solution.f90:33-59), built on the device from the perturbation
    // (launch_init_lattice); the host builds only the edge constants
    auto uv = [&](size_t q, double &u, double &v) {
        u = h->p.uu;
        v = 0.0;
        if (du) u = u + du[q];
        if (dv) v = v + dv[q];
    };
    // edge f0 = the initial f on the four edges (streaming never rewrites
    // them, solution.f90:440-447) and the boundary values taken from them
    std::vector<double> ef(9 * (2 * (size_t)ny + 2 * (size_t)nx));
    auto edge_node = [&](size_t at, int i, int j) {
        double u, v;
        uv((size_t)j * nx + i, u, v);
        for (int k = 0; k < 9; ++k) ef[9 * at + k] = feq(1.0, u, v, k);
    };
    for (int j = 0; j < ny; ++j) {
        edge_node((size_t)j, 0, j);
        edge_node((size_t)ny + j, nx - 1, j);
    }
    for (int i = 0; i < nx; ++i) {
        edge_node(2 * (size_t)ny + i, i, 0);
        edge_node(2 * (size_t)ny + nx + i, i, ny - 1);
    }
    {
        const int rc = handle_set_edges(h, ef.data());
        if (rc) return rc;
    }
    // populations and the initial fields (rho = 1, u, v) in slot 0: u0 of the
    // first step. The perturbation goes up into the second population buffer,
    // which the first step overwrites before anything reads it: 9 planes of
    // at least nx*ny elements of at least 2 bytes hold the 2*nx*ny doubles,
    // and no allocation is needed.
    double *ddu = nullptr, *ddv = nullptr;
    if (du || dv) {
        double *stage = (double *)h->fbuf[1];
        if (du) CK(xfer_h2d(ddu = stage, du, sizeof(double) * nn, h->stream), "copy du");
        if (dv) CK(xfer_h2d(ddv = stage + nn, dv, sizeof(double) * nn, h->stream), "copy dv");
    }
    if (launch_init_lattice(h, ddu, ddv)) return cuda_err(h, cudaGetLastError(), "init");
    h->cur = 0;
    h->fields_slot = 0;
    h->fields_step[0] = 0;
    h->fields_step[1] = -1;
    CK(cudaMemsetAsync(h->d_status, 0, sizeof(unsigned), h->stream), "clear status");
    CK(cudaMemsetAsync(h->d_pinfo, 0, LBM_NSLOT_MAX * sizeof(PatchInfo), h->stream), "clear pinfo");
    CK(cudaStreamSynchronize(h->stream), "sync init");
    h->n = 1;
    h->steps_done = 0;
    // the patch rectangles were cleared above: the factorization slots are
    // filled again from the first step
    forget_batches(h);
    h->inited = 1;
    return LBM_OK;
}

int lbm_step(lbm_t *h, double *force_row)
{
    if (!h) return LBM_ERR_ARG;
    return run_steps(h, 1, force_row, nullptr, true);
}

int lbm_run(lbm_t *h, int nsteps, double *force_rows, int *done_steps)
{
    if (!h) return LBM_ERR_ARG;
    if (done_steps) *done_steps = 0;
    if (nsteps < 0) return set_err(h, LBM_ERR_ARG, "run: negative step count");
    if (nsteps == 0) return LBM_OK;
    return run_steps(h, nsteps, force_rows, done_steps, false);
}

int lbm_force_row_length(const lbm_t *h) { return h ? h->row_len : LBM_ERR_ARG; }

int lbm_get_fields(lbm_t *h, double *rho, double *u, double *v)
{
    if (!h) return LBM_ERR_ARG;
    if (!h->inited) return set_err(h, LBM_ERR_STATE, "get_fields: not initialised");
    const int slot = h->fields_slot;
    if (h->fields_step[slot] != h->steps_done)
        return set_err(h, LBM_ERR_STATE, "get_fields: the last step did not keep its fields");
    const size_t nn = (size_t)h->nx * h->ny;
    double *dst[3] = {rho, u, v};
    for (int c = 0; c < 3; ++c) {
        if (!dst[c]) continue;
        if (h->prec == LBM_PREC_FP64)
            CK(xfer_d2h(dst[c], (const double *)h->d_fields[slot] + c * nn, sizeof(double) * nn, h->stream),
               "copy fields");
        else
            CK(xfer_d2h_widen(dst[c], (const float *)h->d_fields[slot] + c * nn, nn, h->stream), "copy fields");
    }
    return LBM_OK;
}

int lbm_get_populations(lbm_t *h, double *f)
{
    if (!h || !f) return LBM_ERR_ARG;
    if (!h->inited) return set_err(h, LBM_ERR_STATE, "get_populations: not initialised");
    const size_t nn = (size_t)h->nx * h->ny;
    if (!h->d_stage) CK(dmalloc(h, &h->d_stage, sizeof(double) * nn * 9), "alloc stage");
    if (launch_unpack(h, h->fbuf[h->cur], h->d_stage)) return cuda_err(h, cudaGetLastError(), "unpack");
    CK(xfer_d2h(f, h->d_stage, sizeof(double) * nn * 9, h->stream), "copy f");
    free_devp(h->d_stage);
    return LBM_OK;
}

int lbm_set_populations(lbm_t *h, const double *f)
{
    if (!h || !f) return LBM_ERR_ARG;
    quiesce(h);   // queued work may still read what is rewritten below
    if (!h->inited) return set_err(h, LBM_ERR_STATE, "set_populations: not initialised");
    const size_t nn = (size_t)h->nx * h->ny;
    if (!h->d_stage) CK(dmalloc(h, &h->d_stage, sizeof(double) * nn * 9), "alloc stage");
    CK(xfer_h2d(h->d_stage, f, sizeof(double) * nn * 9, h->stream), "copy f");
    if (launch_pack(h, h->d_stage, h->fbuf[h->cur])) return cuda_err(h, cudaGetLastError(), "pack");
    CK(cudaStreamSynchronize(h->stream), "sync f");
    free_devp(h->d_stage);
    h->fields_step[0] = h->fields_step[1] = -1;
    return LBM_OK;
}

int lbm_residual(lbm_t *h, double *err)
{
    if (!h || !err) return LBM_ERR_ARG;
    const int a = h->fields_slot, b = a ^ 1;
    if (h->steps_done < 1 || h->fields_step[a] != h->steps_done || h->fields_step[b] != h->steps_done - 1)
        return set_err(h, LBM_ERR_STATE, "residual: fields of the last two states were not kept");
    double s[2];
    if (launch_residual(h, h->d_fields[a], h->d_fields[b], s)) return cuda_err(h, cudaGetLastError(), "residual");
    *err = sqrt(s[0]) / (sqrt(s[1]) + 1e-30);   // solution.f90:120-122
    return LBM_OK;
}

int lbm_mass(lbm_t *h, double *mass)
{
    if (!h || !mass) return LBM_ERR_ARG;
    if (!h->inited) return set_err(h, LBM_ERR_STATE, "mass: not initialised");
    if (launch_mass(h, h->fbuf[h->cur], h->stream)) return cuda_err(h, cudaGetLastError(), "launch mass");
    CK(cudaMemcpyAsync(h->hblock, h->d_head, sizeof(RunHead), cudaMemcpyDeviceToHost, h->stream), "copy mass");
    CK(cudaStreamSynchronize(h->stream), "sync mass");
    const int rc = mass_result(h, ((const RunHead *)h->hblock)->mass);
    *mass = h->last_mass;
    return rc;
}

int lbm_get_markers(lbm_t *h, double *xb2, double *yb2, double *solve_residual, int *half_bandwidth)
{
    if (!h) return LBM_ERR_ARG;
    if (!h->ib_ready || h->nseg == 0) return set_err(h, LBM_ERR_STATE, "get_markers: no immersed boundary step run");
    std::vector<Marker> mk(h->nseg);
    const Marker *last = h->d_mk + (size_t)((h->n - 1) % h->nslots) * h->nseg;   // slot of the last step
    CK(cudaMemcpyAsync(mk.data(), last, sizeof(Marker) * h->nseg, cudaMemcpyDeviceToHost, h->stream), "copy markers");
    double res[2] = {0, 0};
    const double *last_res = h->d_solve_res + 2 * ((h->n - 1) % h->nslots);
    CK(cudaMemcpyAsync(res, last_res, 2 * sizeof(double), cudaMemcpyDeviceToHost, h->stream), "copy res");
    CK(cudaStreamSynchronize(h->stream), "sync markers");
    for (int k = 0; k < h->nseg; ++k) {
        if (xb2) xb2[k] = mk[k].xm;
        if (yb2) yb2[k] = mk[k].ym;
    }
    if (solve_residual) *solve_residual = res[0];
    if (half_bandwidth) *half_bandwidth = (int)res[1];
    return LBM_OK;
}

int lbm_set_timing(lbm_t *h, int enable)
{
    if (!h) return LBM_ERR_ARG;
    if (enable && h->ev.empty()) {
        h->ev.resize(4 * (size_t)h->ring_cap);
        h->ev_side.resize(2 * (size_t)h->ring_cap);
        for (auto &e : h->ev) CK(cudaEventCreate(&e), "event create");
        for (auto &e : h->ev_side) CK(cudaEventCreate(&e), "event create");
    }
    h->timing = enable == LBM_TIMING_SPAN ? LBM_TIMING_SPAN : (enable ? LBM_TIMING_KERNELS : 0);
    h->t_step = h->t_ib = h->t_kf = 0;
    h->t_steps = 0;
    return LBM_OK;
}

int lbm_get_timing(lbm_t *h, double *step_ms, double *ib_ms, double *lattice_ms, int *steps)
{
    if (!h) return LBM_ERR_ARG;
    if (step_ms) *step_ms = h->t_step;
    if (ib_ms) *ib_ms = h->t_ib;
    if (lattice_ms) *lattice_ms = h->t_kf;
    if (steps) *steps = h->t_steps;
    return LBM_OK;
}

int lbm_get_launch_count(const lbm_t *h, long long *count)
{
    if (!h || !count) return LBM_ERR_ARG;
    *count = h->launches;
    return LBM_OK;
}

int lbm_get_device_launches(const lbm_t *h, long long *count)
{
    if (!h || !count) return LBM_ERR_ARG;
    *count = h->device_launches;
    return LBM_OK;
}

int lbm_step_index(const lbm_t *h) { return h ? h->n : LBM_ERR_ARG; }

int lbm_device_bytes(const lbm_t *h, long long *bytes)
{
    if (!h || !bytes) return LBM_ERR_ARG;
    *bytes = h->dev_bytes;
    return LBM_OK;
}

const char *lbm_last_error(const lbm_t *h) { return h ? h->err.c_str() : "lbm_create failed (bad parameters or no CUDA device)"; }

int lbm_device_check(int *binary_version, int *sm_count)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return LBM_ERR_CUDA;
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, arch_probe) != cudaSuccess) return LBM_ERR_CUDA;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return LBM_ERR_CUDA;
    if (binary_version) *binary_version = fa.binaryVersion;
    if (sm_count) *sm_count = sms;
    return LBM_OK;
}

int lbm_describe_status(unsigned int status, char *message, int capacity)
{
    std::string msg;
    const int code = status_error(status, msg);
    if (message && capacity > 0) {
        const size_t n = std::min(msg.size(), (size_t)capacity - 1);
        memcpy(message, msg.data(), n);
        message[n] = 0;
    }
    return code;
}

}  // extern "C"
