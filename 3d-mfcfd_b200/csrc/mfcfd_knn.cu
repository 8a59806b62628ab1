/*
 * mfcfd_knn.cu - k nearest neighbours of every point of a cloud
 * (mfcfd_knn), the connectivity a cloud without one needs before the
 * reference's set-up can run (the reference reads conn from its input file,
 * point_preprocessor.f90:30-35; a request server must build it).
 *
 * The answer is defined exactly, so the GPU and the host give the same
 * arrays: the neighbours of point i are the k points j != i with the
 * smallest (d2, j), where d2 = dx*dx + dy*dy + dz*dz with dx = x[j] - x[i]
 * (evaluated in that order, without contraction), listed in that order;
 * min_dist is sqrt(d2) of the first.  Two points at distance 0 are an
 * error.
 *
 * Search structure: the points sorted along a Morton curve, cut into leaves
 * of KNN_LEAF consecutive points, with levels of nodes over KNN_FAN
 * consecutive children, each carrying its points' bounding box.  A query
 * first takes its own leaf, then walks the tree depth first, skipping every
 * node whose box lies farther than its current k-th distance (with a
 * relative margin far above rounding, so no candidate is ever skipped).
 * The host's walk is knn_query (a pool of threads), the device's k_knn_query
 * (a warp per query).
 */
#include <cuda_runtime.h>
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <exception>
#include <string>
#include <thread>
#include <vector>

#include "mfcfd_internal.h"

namespace mfcfd {
namespace {

constexpr int KNN_LEAF = 32;
constexpr int KNN_FAN = 8;
constexpr int KNN_MAX_LEVELS = 16;
constexpr int KNN_STACK = KNN_MAX_LEVELS * KNN_FAN;
constexpr double KNN_MARGIN = 1.0 + 1e-9;

struct Box6 {
    double lo[3], hi[3];
};

// The tree over the sorted points: level 0 are the leaves (KNN_LEAF points
// each), level l+1 groups KNN_FAN nodes of level l; node b of level l
// covers the sorted points [b * span_l, min(n, (b+1) * span_l)).
struct KnnTree {
    int n = 0, levels = 0;
    int count[KNN_MAX_LEVELS];
    long long span[KNN_MAX_LEVELS];
    const Box6 *box[KNN_MAX_LEVELS];
    const double *sx, *sy, *sz;   // coordinates in sorted order
    const int32_t *id;            // sorted position -> point index
};

__host__ __device__ inline int min_i(int a, int b) { return a < b ? a : b; }

__host__ __device__ inline double box_d2(const Box6 &b, double px, double py, double pz) {
    const double p[3] = {px, py, pz};
    double s = 0.0;
    for (int a = 0; a < 3; ++a) {
        const double d = p[a] < b.lo[a] ? b.lo[a] - p[a] : (p[a] > b.hi[a] ? p[a] - b.hi[a] : 0.0);
        s = s + d * d;
    }
    return s;
}

// insert (d2, j) into the ascending list (bd, bj) of length *m <= k
inline void knn_insert(double d2, int j, double *bd, int *bj, int *m, int k) {
    int at = *m;
    if (at == k) {
        if (!(d2 < bd[k - 1] || (d2 == bd[k - 1] && j < bj[k - 1]))) return;
        at = k - 1;
    } else {
        ++*m;
    }
    while (at > 0 && (d2 < bd[at - 1] || (d2 == bd[at - 1] && j < bj[at - 1]))) {
        bd[at] = bd[at - 1];
        bj[at] = bj[at - 1];
        --at;
    }
    bd[at] = d2;
    bj[at] = j;
}

// the k nearest neighbours of sorted point q (bd, bj ascending; returns how
// many were found, < k only when the cloud has fewer than k + 1 points);
// *dup is set when another point coincides with it
inline int knn_query(const KnnTree &t, int q, int k, double *bd, int *bj, int *dup) {
    const double px = t.sx[q], py = t.sy[q], pz = t.sz[q];
    const int self = t.id[q];
    int m = 0;
    auto scan_leaf = [&](int leaf) {
        const int a = leaf * KNN_LEAF, b = min_i(t.n, a + KNN_LEAF);
        for (int s = a; s < b; ++s) {
            const int j = t.id[s];
            if (j == self) continue;
            const double dx = t.sx[s] - px, dy = t.sy[s] - py, dz = t.sz[s] - pz;
            const double d2 = dx * dx + dy * dy + dz * dz;
            if (d2 == 0.0) *dup = 1;
            knn_insert(d2, j, bd, bj, &m, k);
        }
    };
    const int own = q / KNN_LEAF;
    scan_leaf(own);
    // depth-first over the tree from the root, nearer children first
    int stack_lvl[KNN_STACK], stack_node[KNN_STACK];
    int sp = 0;
    stack_lvl[sp] = t.levels - 1;
    stack_node[sp] = 0;
    ++sp;
    while (sp > 0) {
        --sp;
        const int l = stack_lvl[sp], b = stack_node[sp];
        const double lim = m == k ? bd[k - 1] * KNN_MARGIN : 1e300;
        if (box_d2(t.box[l][b], px, py, pz) > lim) continue;
        if (l == 0) {
            if (b != own) scan_leaf(b);
            continue;
        }
        // children of b at level l-1, pushed farthest first
        const int c0 = b * KNN_FAN, c1 = min_i(t.count[l - 1], c0 + KNN_FAN);
        double cd[KNN_FAN];
        int ci[KNN_FAN], nc = 0;
        for (int c = c0; c < c1; ++c) {
            const double dd = box_d2(t.box[l - 1][c], px, py, pz);
            if (dd > lim) continue;
            int at = nc++;
            while (at > 0 && cd[at - 1] < dd) {   // descending distance
                cd[at] = cd[at - 1];
                ci[at] = ci[at - 1];
                --at;
            }
            cd[at] = dd;
            ci[at] = c;
        }
        for (int c = 0; c < nc && sp < KNN_STACK; ++c) {
            stack_lvl[sp] = l - 1;
            stack_node[sp] = ci[c];
            ++sp;
        }
    }
    return m;
}


__host__ __device__ inline uint64_t knn_spread3(uint64_t v) {
    v &= 0x1fffffull;
    v = (v | (v << 32)) & 0x1f00000000ffffull;
    v = (v | (v << 16)) & 0x1f0000ff0000ffull;
    v = (v | (v << 8)) & 0x100f00f00f00f00full;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

__host__ __device__ inline uint64_t knn_key(double x, double y, double z, const double *lo, const double *scale) {
    const double v[3] = {x, y, z};
    uint64_t q[3];
    for (int a = 0; a < 3; ++a) {
        double u = (v[a] - lo[a]) * scale[a];
        u = u < 0.0 ? 0.0 : (u > 2097151.0 ? 2097151.0 : u);
        q[a] = (uint64_t)u;
    }
    return knn_spread3(q[0]) | (knn_spread3(q[1]) << 1) | (knn_spread3(q[2]) << 2);
}

// the box of node b of a level from its range of sorted points (level 0) or
// its children's boxes
__host__ __device__ inline Box6 knn_leaf_box(int b, int n, const double *sx, const double *sy, const double *sz) {
    Box6 r;
    const int a = b * KNN_LEAF, e = min_i(n, a + KNN_LEAF);
    r.lo[0] = r.hi[0] = sx[a];
    r.lo[1] = r.hi[1] = sy[a];
    r.lo[2] = r.hi[2] = sz[a];
    for (int s = a + 1; s < e; ++s) {
        const double v[3] = {sx[s], sy[s], sz[s]};
        for (int k = 0; k < 3; ++k) {
            r.lo[k] = v[k] < r.lo[k] ? v[k] : r.lo[k];
            r.hi[k] = v[k] > r.hi[k] ? v[k] : r.hi[k];
        }
    }
    return r;
}

__host__ __device__ inline Box6 knn_node_box(int b, int nchild, const Box6 *child) {
    const int a = b * KNN_FAN, e = min_i(nchild, a + KNN_FAN);
    Box6 r = child[a];
    for (int c = a + 1; c < e; ++c)
        for (int k = 0; k < 3; ++k) {
            r.lo[k] = child[c].lo[k] < r.lo[k] ? child[c].lo[k] : r.lo[k];
            r.hi[k] = child[c].hi[k] > r.hi[k] ? child[c].hi[k] : r.hi[k];
        }
    return r;
}

// one query's output rows (conn 1-based, zero padded to MAX_CONN)
inline void knn_store(const KnnTree &t, int q, int k, int32_t *nbhs, int32_t *conn,
                                          double *min_dist, int *dup, int *short_) {
    double bd[MAX_CONN];
    int bj[MAX_CONN];
    const int m = knn_query(t, q, k, bd, bj, dup);
    const int i = t.id[q];
    if (m < k) *short_ = 1;
    nbhs[i] = m;
    for (int r = 0; r < MAX_CONN; ++r) conn[(size_t)i * MAX_CONN + r] = r < m ? bj[r] + 1 : 0;
    min_dist[i] = m > 0 ? sqrt(bd[0]) : 0.0;
}

__global__ void k_knn_keys(int n, const double *x, const double *y, const double *z, Box6 b, uint64_t *key,
                           int32_t *idx) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    key[i] = knn_key(x[i], y[i], z[i], b.lo, b.hi);   // hi carries the scale
    idx[i] = i;
}

__global__ void k_knn_gather(int n, const int32_t *id, const double *x, const double *y, const double *z,
                             double *sx, double *sy, double *sz) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    sx[s] = x[id[s]];
    sy[s] = y[id[s]];
    sz[s] = z[id[s]];
}

__global__ void k_knn_leaves(int count, int n, const double *sx, const double *sy, const double *sz, Box6 *box) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < count) box[b] = knn_leaf_box(b, n, sx, sy, sz);
}

__global__ void k_knn_nodes(int count, int nchild, const Box6 *child, Box6 *box) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < count) box[b] = knn_node_box(b, nchild, child);
}

// (d, j) before (e, i) in the neighbours' order
__device__ __forceinline__ bool knn_before(double d, int j, double e, int i) { return d < e || (d == e && j < i); }

// Squared distance of sorted point s to the query; a NaN counts as farthest.
__device__ __forceinline__ double knn_d2(const KnnTree &t, int s, double px, double py, double pz) {
    const double dx = t.sx[s] - px, dy = t.sy[s] - py, dz = t.sz[s] - pz;
    const double d2 = dx * dx + dy * dy + dz * dz;
    return d2 == d2 ? d2 : INFINITY;
}

// A warp per query, neighbouring queries in neighbouring warps: lane r holds
// the r-th nearest so far (k <= 27 of the 32 are read), a leaf's points are
// tested a lane each and the few nearer than the k-th are inserted by a shift
// across the lanes; a node's children are ranked by distance a lane each onto
// a stack in shared memory.  The point's own leaf is sorted by a bitonic
// network.  Bound by the shuffles' latency and issue; a thread per query kept
// its list and stack in local memory and diverged at each insertion (250,620
// points, k = 26: 12.7 ms against 2.5).
constexpr int KNN_WARPS = 4;
__global__ void __launch_bounds__(KNN_WARPS * 32) k_knn_query(const __grid_constant__ KnnTree t, int k, int32_t *nbhs,
                                                              int32_t *conn, double *min_dist, int *flags) {
    static_assert(KNN_LEAF == 32 && KNN_FAN <= 32 && MAX_CONN <= 32, "a lane per leaf point, child and neighbour");
    constexpr unsigned ALL = 0xffffffffu;
    __shared__ double stack_d[KNN_WARPS][KNN_STACK];
    __shared__ int2 stack_n[KNN_WARPS][KNN_STACK];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = blockIdx.x * KNN_WARPS + warp;
    if (q >= t.n) return;
    double *sd = stack_d[warp];
    int2 *sn = stack_n[warp];
    const double px = t.sx[q], py = t.sy[q], pz = t.sz[q];
    const int own = q / KNN_LEAF;
    bool dup = false;
    double bd = INFINITY;
    int bj = INT_MAX;
    if (own * KNN_LEAF + lane < t.n && own * KNN_LEAF + lane != q) {
        bd = knn_d2(t, own * KNN_LEAF + lane, px, py, pz);
        bj = t.id[own * KNN_LEAF + lane];
        dup = bd == 0.0;
    }
#pragma unroll
    for (int size = 2; size <= 32; size *= 2)
#pragma unroll
        for (int step = size / 2; step > 0; step /= 2) {
            const double od = __shfl_xor_sync(ALL, bd, step);
            const int oj = __shfl_xor_sync(ALL, bj, step);
            const bool first = ((lane & step) == 0) == ((lane & size) == 0);   // keeps the nearer of the two
            if (knn_before(od, oj, bd, bj) == first) {
                bd = od;
                bj = oj;
            }
        }
    double kd = __shfl_sync(ALL, bd, k - 1);
    int kj = __shfl_sync(ALL, bj, k - 1);
    int sp = 0;
    if (lane == 0) {
        sd[0] = 0.0;
        sn[0] = make_int2(t.levels - 1, 0);
    }
    sp = 1;
    __syncwarp();
    while (sp > 0) {
        --sp;
        const double dist = sd[sp];
        const int l = sn[sp].x, b = sn[sp].y;
        __syncwarp();                                   // read before the slot is written again
        const double lim = kj != INT_MAX ? kd * KNN_MARGIN : 1e300;
        if (dist > lim) continue;
        if (l > 0) {
            // the children within reach, farthest first (the nearest on top)
            const int c = b * KNN_FAN + lane;
            const bool valid = lane < KNN_FAN && c < t.count[l - 1];
            const double dd = valid ? box_d2(t.box[l - 1][c], px, py, pz) : 0.0;
            const bool in = valid && !(dd > lim);
            const unsigned mask = __ballot_sync(ALL, in);
            int at = sp;
#pragma unroll
            for (int r = 0; r < KNN_FAN; ++r) {
                const double od = __shfl_sync(ALL, dd, r);
                if ((mask >> r & 1u) && (od > dd || (od == dd && r < lane))) ++at;
            }
            if (in) {
                sd[at] = dd;
                sn[at] = make_int2(l - 1, c);
            }
            sp += __popc(mask);
            __syncwarp();
            continue;
        }
        if (b == own) continue;
        const int s = b * KNN_LEAF + lane;
        double d = INFINITY;
        int j = INT_MAX;
        if (s < t.n) {
            d = knn_d2(t, s, px, py, pz);
            j = t.id[s];
            dup = dup || d == 0.0;
        }
        for (unsigned near = __ballot_sync(ALL, knn_before(d, j, kd, kj)); near; near &= near - 1u) {
            const int src = __ffs(near) - 1;
            const double cd = __shfl_sync(ALL, d, src);
            const int cj = __shfl_sync(ALL, j, src);
            if (!knn_before(cd, cj, kd, kj)) continue;
            const int rank = __popc(__ballot_sync(ALL, knn_before(bd, bj, cd, cj)));
            const double ud = __shfl_up_sync(ALL, bd, 1);
            const int uj = __shfl_up_sync(ALL, bj, 1);
            if (lane >= rank) {
                bd = lane == rank ? cd : ud;
                bj = lane == rank ? cj : uj;
            }
            kd = __shfl_sync(ALL, bd, k - 1);
            kj = __shfl_sync(ALL, bj, k - 1);
        }
    }
    const int i = t.id[q];
    const bool have = lane < k && bj != INT_MAX;
    const int m = __popc(__ballot_sync(ALL, have));
    if (lane < MAX_CONN) conn[(size_t)i * MAX_CONN + lane] = have ? bj + 1 : 0;   // 1-based, zero padded
    if (__any_sync(ALL, dup) && lane == 0) atomicExch(&flags[0], 1);
    if (lane == 0) {
        nbhs[i] = m;
        min_dist[i] = m > 0 ? sqrt(bd) : 0.0;
        if (m < k) atomicExch(&flags[1], 1);
    }
}

// bounding box and Morton scale over the cloud (exact minima and maxima)
void knn_frame(int n, const double *x, const double *y, const double *z, double lo[3], double scale[3]) {
    double hi[3] = {x[0], y[0], z[0]};
    lo[0] = x[0]; lo[1] = y[0]; lo[2] = z[0];
    for (int i = 1; i < n; ++i) {
        const double v[3] = {x[i], y[i], z[i]};
        for (int a = 0; a < 3; ++a) {
            lo[a] = std::min(lo[a], v[a]);
            hi[a] = std::max(hi[a], v[a]);
        }
    }
    for (int a = 0; a < 3; ++a) scale[a] = hi[a] > lo[a] ? 2097151.0 / (hi[a] - lo[a]) : 0.0;
}

int level_counts(int n, int count[KNN_MAX_LEVELS], long long span[KNN_MAX_LEVELS]) {
    int levels = 0;
    long long sp = KNN_LEAF;
    int c = (n + KNN_LEAF - 1) / KNN_LEAF;
    while (true) {
        count[levels] = c;
        span[levels] = sp;
        ++levels;
        if (c == 1 || levels == KNN_MAX_LEVELS) break;
        c = (c + KNN_FAN - 1) / KNN_FAN;
        sp *= KNN_FAN;
    }
    return levels;
}

// stream-ordered scratch, so a search beside running solves does not wait
// for the whole device
struct KnnBufs {
    std::vector<void *> p;
    cudaStream_t s;
    explicit KnnBufs(cudaStream_t st) : s(st) {}
    ~KnnBufs() {
        for (void *v : p) cudaFreeAsync(v, s);
        cudaStreamSynchronize(s);
    }
    template <typename T>
    cudaError_t alloc(T **ptr, size_t count) {
        void *v = nullptr;
        cudaError_t e = cudaMallocAsync(&v, sizeof(T) * (count ? count : 1), s);
        if (e == cudaSuccess) p.push_back(v);
        *ptr = (T *)v;
        return e;
    }
};

#define KNN_CK(call)                                                   \
    do {                                                               \
        cudaError_t e_ = (call);                                       \
        if (e_ != cudaSuccess) {                                       \
            err = std::string(#call) + ": " + cudaGetErrorString(e_);  \
            return e_ == cudaErrorMemoryAllocation ? MFCFD_ERR_NOMEM : MFCFD_ERR_CUDA; \
        }                                                              \
    } while (0)

int knn_device(int device, int n, const double *x, const double *y, const double *z, int k, int32_t *nbhs,
               int32_t *conn, double *min_dist, std::string &err) {
    KNN_CK(cudaSetDevice(device));
    cudaStream_t s = nullptr;
    KNN_CK(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    struct StreamGuard {
        cudaStream_t s;
        ~StreamGuard() { cudaStreamDestroy(s); }
    } guard{s};
    KnnBufs b(s);
    double *dx, *dy, *dz, *sx, *sy, *sz, *dmd;
    uint64_t *key, *key2;
    int32_t *idx, *id, *dnb, *dconn;
    int *flags;
    KNN_CK(b.alloc(&dx, n)); KNN_CK(b.alloc(&dy, n)); KNN_CK(b.alloc(&dz, n));
    KNN_CK(b.alloc(&sx, n)); KNN_CK(b.alloc(&sy, n)); KNN_CK(b.alloc(&sz, n));
    KNN_CK(b.alloc(&key, n)); KNN_CK(b.alloc(&key2, n)); KNN_CK(b.alloc(&idx, n)); KNN_CK(b.alloc(&id, n));
    KNN_CK(b.alloc(&dnb, n)); KNN_CK(b.alloc(&dconn, (size_t)n * MAX_CONN)); KNN_CK(b.alloc(&dmd, n));
    KNN_CK(b.alloc(&flags, 2));
    KNN_CK(cudaMemcpyAsync(dx, x, 8 * (size_t)n, cudaMemcpyHostToDevice, s));
    KNN_CK(cudaMemcpyAsync(dy, y, 8 * (size_t)n, cudaMemcpyHostToDevice, s));
    KNN_CK(cudaMemcpyAsync(dz, z, 8 * (size_t)n, cudaMemcpyHostToDevice, s));
    KNN_CK(cudaMemsetAsync(flags, 0, 2 * sizeof(int), s));
    Box6 fr;
    knn_frame(n, x, y, z, fr.lo, fr.hi);
    const int T = 256, g = (n + T - 1) / T;
    k_knn_keys<<<g, T, 0, s>>>(n, dx, dy, dz, fr, key, idx);
    size_t bytes = 0;
    KNN_CK(cub::DeviceRadixSort::SortPairs(nullptr, bytes, key, key2, idx, id, n, 0, 64, s));
    uint8_t *scratch;
    KNN_CK(b.alloc(&scratch, bytes));
    KNN_CK(cub::DeviceRadixSort::SortPairs(scratch, bytes, key, key2, idx, id, n, 0, 64, s));
    k_knn_gather<<<g, T, 0, s>>>(n, id, dx, dy, dz, sx, sy, sz);
    KnnTree t;
    t.n = n;
    t.levels = level_counts(n, t.count, t.span);
    Box6 *boxes[KNN_MAX_LEVELS];
    for (int l = 0; l < t.levels; ++l) {
        KNN_CK(b.alloc(&boxes[l], t.count[l]));
        const int gl = (t.count[l] + T - 1) / T;
        if (l == 0) k_knn_leaves<<<gl, T, 0, s>>>(t.count[0], n, sx, sy, sz, boxes[0]);
        else k_knn_nodes<<<gl, T, 0, s>>>(t.count[l], t.count[l - 1], boxes[l - 1], boxes[l]);
        t.box[l] = boxes[l];
    }
    t.sx = sx; t.sy = sy; t.sz = sz; t.id = id;
    k_knn_query<<<(n + KNN_WARPS - 1) / KNN_WARPS, KNN_WARPS * 32, 0, s>>>(t, k, dnb, dconn, dmd, flags);
    KNN_CK(cudaGetLastError());
    int h_flags[2] = {0, 0};
    KNN_CK(cudaMemcpyAsync(h_flags, flags, sizeof h_flags, cudaMemcpyDeviceToHost, s));
    KNN_CK(cudaMemcpyAsync(nbhs, dnb, 4 * (size_t)n, cudaMemcpyDeviceToHost, s));
    KNN_CK(cudaMemcpyAsync(conn, dconn, 4 * (size_t)n * MAX_CONN, cudaMemcpyDeviceToHost, s));
    KNN_CK(cudaMemcpyAsync(min_dist, dmd, 8 * (size_t)n, cudaMemcpyDeviceToHost, s));
    KNN_CK(cudaStreamSynchronize(s));
    if (h_flags[0]) {
        err = "two points of the cloud coincide";
        return MFCFD_ERR_ARG;
    }
    if (h_flags[1]) {
        err = "the cloud has no more than k points";
        return MFCFD_ERR_ARG;
    }
    return MFCFD_OK;
}

int knn_host(int n, const double *x, const double *y, const double *z, int k, int32_t *nbhs, int32_t *conn,
             double *min_dist, std::string &err) {
    double lo[3], scale[3];
    knn_frame(n, x, y, z, lo, scale);
    std::vector<std::pair<uint64_t, int32_t>> key(n);
    for (int i = 0; i < n; ++i) key[i] = {knn_key(x[i], y[i], z[i], lo, scale), i};
    std::sort(key.begin(), key.end());
    std::vector<int32_t> id(n);
    std::vector<double> sx(n), sy(n), sz(n);
    for (int s = 0; s < n; ++s) {
        id[s] = key[s].second;
        sx[s] = x[id[s]];
        sy[s] = y[id[s]];
        sz[s] = z[id[s]];
    }
    KnnTree t;
    t.n = n;
    t.levels = level_counts(n, t.count, t.span);
    std::vector<Box6> boxes[KNN_MAX_LEVELS];
    for (int l = 0; l < t.levels; ++l) {
        boxes[l].resize(t.count[l]);
        for (int b = 0; b < t.count[l]; ++b)
            boxes[l][b] = l == 0 ? knn_leaf_box(b, n, sx.data(), sy.data(), sz.data())
                                 : knn_node_box(b, t.count[l - 1], boxes[l - 1].data());
        t.box[l] = boxes[l].data();
    }
    t.sx = sx.data(); t.sy = sy.data(); t.sz = sz.data(); t.id = id.data();
    // the queries on the calling thread and the set-up pool's threads
    const int want = std::min(31, n / 4096);
    const int extra = want > 0 ? take_setup_threads(want) : 0;
    const int nt = extra + 1;
    std::vector<int> dup(nt, 0), sh(nt, 0);
    auto run = [&](int w) {
        for (int q = w; q < n; q += nt) knn_store(t, q, k, nbhs, conn, min_dist, &dup[w], &sh[w]);
    };
    std::vector<std::thread> th;
    std::exception_ptr e0;
    try {
        for (int w = 1; w < nt; ++w) th.emplace_back(run, w);
    } catch (...) {
        e0 = std::current_exception();
    }
    if (!e0) run(0);
    for (auto &h : th) h.join();
    give_setup_threads(extra);
    if (e0) std::rethrow_exception(e0);
    for (int w = 0; w < nt; ++w) {
        if (dup[w]) {
            err = "two points of the cloud coincide";
            return MFCFD_ERR_ARG;
        }
        if (sh[w]) {
            err = "the cloud has no more than k points";
            return MFCFD_ERR_ARG;
        }
    }
    return MFCFD_OK;
}

}  // namespace

int knn_connectivity(int device, int n, const double *x, const double *y, const double *z, int k, int32_t *nbhs,
                     int32_t *conn, double *min_dist, std::string &err) {
    if (n < 1 || k < 1 || k > MAX_CONN) {
        err = "knn: need n >= 1 and 1 <= k <= 27";
        return MFCFD_ERR_ARG;
    }
    return device >= 0 ? knn_device(device, n, x, y, z, k, nbhs, conn, min_dist, err)
                       : knn_host(n, x, y, z, k, nbhs, conn, min_dist, err);
}

}  // namespace mfcfd
