// Euclidean clustering on the GPU: the radius search and cluster extraction of
// DAPHNE's euclidean_cluster kernel (extractEuclideanClusters / extract,
// src/CPU/euclidean_cluster/kernel.cpp:562-647; its CUDA port builds an N x N
// boolean distance matrix, src/Cuda/euclidean_cluster/kernel.cu:506-560), and
// the host side of segmentByDistance / clusterAndColor (:652-814) around it.
//
// The reference grows each cluster breadth-first from its smallest
// unprocessed point through all points whose float squared distance
// dx*dx + dy*dy + dz*dz (each product and sum rounded) is <= r*r (float): the
// clusters are the connected components of that graph, in order of their
// smallest point index, each listed in ascending index order; those with
// [min, max] points are kept and ordered by size with std::sort over reverse
// iterators.
//
// Here the points of all distance rings of up to 8 clouds go through one pass:
// a kernel finds every point's part (cloud and ring) and the parts' bounding
// boxes; points are sorted into cells of edge r * (1 + 1e-4) of their part
// (cell indices in FP64, so an accepted pair is never more than one cell apart
// on any axis; at most 2^28 cells in all) with the voxel-grid build's stable
// radix sort; a warp per point tests the earlier points of its own and the
// neighbour cells with the same float operations.  A first pass hangs every
// point under the first one it is joined to, a second joins the trees in a
// lock-free union-find (the larger root is linked under the smaller by
// atomicCAS); every label is its tree's smallest point index.  A second sort, by
// label, lists the clusters: in the reference's order, their points ascending.
// The host applies the same std::sort to the sizes and spreads the clusters'
// points, centroids and boxes over its threads.
#include <cuda_runtime.h>
#include <stdint.h>

#include <limits.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <string>
#include <vector>

#include "../../include/ndt_b200.h"
#include "ec_pose.h"
#include "grid_build.h"
#include "nvtx_range.h"

namespace ec {

constexpr int kThreads = 256;
constexpr unsigned kAll = 0xffffffffu;
constexpr int kUnionLimit = 1 << 20;  // CAS retries of one union (never reached in practice; flags an error)

constexpr int kMaxParts = 40;  // parts clustered in one pass (segmentByDistance: 5 rings of up to 8 clouds)

// Geometry of the parts of one pass: part p's cells have edge cell[p] from
// minv[p] with dims dim[p], and its cell keys are base[p] + x + dx (y + dy z).
struct Parts {
    long long base[kMaxParts + 1];
    float minv[kMaxParts][3];
    float cell[kMaxParts];
    float r2[kMaxParts];
    int dim[kMaxParts][3];
};

// Which part a point belongs to: the distance ring of its cloud, or one part
// for all (rings == 1).
constexpr int kRings = 5;
struct Clouds {
    int count, rings;
    int off[kMaxParts / kRings + 1];
};
__host__ __device__ inline int ring_of(float x, float y) {
    const float d = sqrtf(x * x + y * y);
    return d < 15 ? 0 : (d < 30 ? 1 : (d < 45 ? 2 : (d < 60 ? 3 : 4)));
}

// A part's bounding box: the coordinates as integers of the same order.
struct Box {
    int lo[3], hi[3];
    int points, bad;  // any points, any coordinate that is not finite
};
__host__ __device__ inline int ordered(int bits) { return bits ^ ((bits >> 31) & 0x7fffffff); }

// Cell index in FP64 (the difference of two floats is exact there), so that
// cell boundaries move by no more than ~1e-16 cells: with cells 1e-4 wider
// than the radius, points of an accepted pair are at most one cell apart.
__device__ __forceinline__ int cell_of(float v, float minv, float cell, int dim) {
    int c = (int)(((double)v - (double)minv) / (double)cell);
    return c < 0 ? 0 : (c >= dim ? dim - 1 : c);
}

// The cloud of point t: the last c with off[c] <= t.
__host__ __device__ inline int cloud_of(const Clouds &C, int t) {
    int lo = 0, hi = C.count;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (C.off[mid] <= t) lo = mid; else hi = mid;
    }
    return lo;
}

// The points as float4 with their part in w, and the parts' boxes (lo starts at
// INT_MAX, hi at INT_MIN).  A warp holds points of few parts: one reduction for
// each of them, then the block's boxes in shared memory.
__global__ void __launch_bounds__(kThreads) part_kernel(const float *__restrict__ xyz, int n,
                                                        const __grid_constant__ Clouds C, float4 *__restrict__ pts,
                                                        Box *__restrict__ boxes) {
    __shared__ Box s_box[kMaxParts];
    const int np = C.count * C.rings;
    for (int k = threadIdx.x; k < np; k += kThreads)
        s_box[k] = {{INT_MAX, INT_MAX, INT_MAX}, {INT_MIN, INT_MIN, INT_MIN}, 0, 0};
    __syncthreads();
    const int i = blockIdx.x * kThreads + threadIdx.x;
    int q = -1, v[3] = {0, 0, 0};
    bool bad = false;
    if (i < n) {
        const float x = xyz[3 * (size_t)i], y = xyz[3 * (size_t)i + 1], z = xyz[3 * (size_t)i + 2];
        q = C.rings * cloud_of(C, i) + (C.rings > 1 ? ring_of(x, y) : 0);
        bad = !(isfinite(x) && isfinite(y) && isfinite(z));
        pts[i] = make_float4(x, y, z, __int_as_float(q));
        v[0] = ordered(__float_as_int(x));
        v[1] = ordered(__float_as_int(y));
        v[2] = ordered(__float_as_int(z));
    }
    for (unsigned left = __ballot_sync(kAll, q >= 0); left;) {
        const int part = __shfl_sync(kAll, q, __ffs(left) - 1);
        const unsigned same = __ballot_sync(kAll, q == part);
        left &= ~same;
        if (q == part) {
            const bool any_bad = __any_sync(same, bad);
            const bool leader = (threadIdx.x & 31) == __ffs(same) - 1;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int lo = __reduce_min_sync(same, v[k]), hi = __reduce_max_sync(same, v[k]);
                if (leader) {
                    atomicMin(&s_box[part].lo[k], lo);
                    atomicMax(&s_box[part].hi[k], hi);
                }
            }
            if (leader) {
                s_box[part].points = 1;
                if (any_bad) s_box[part].bad = 1;
            }
        }
        __syncwarp();
    }
    __syncthreads();
    for (int k = threadIdx.x; k < 6 * np; k += kThreads) {
        const int part = k / 6, c = k % 6;
        if (!s_box[part].points) continue;
        if (c < 3) atomicMin(&boxes[part].lo[c], s_box[part].lo[c]);
        else atomicMax(&boxes[part].hi[c - 3], s_box[part].hi[c - 3]);
        if (c == 0) boxes[part].points = 1;
        if (c == 0 && s_box[part].bad) boxes[part].bad = 1;
    }
}

__global__ void key_kernel(const float4 *__restrict__ pts, int n, const __grid_constant__ Parts P,
                           uint32_t *__restrict__ keys, int *__restrict__ least) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = pts[i];
    const int q = __float_as_int(p.w);
    const int cx = cell_of(p.x, P.minv[q][0], P.cell[q], P.dim[q][0]);
    const int cy = cell_of(p.y, P.minv[q][1], P.cell[q], P.dim[q][1]);
    const int cz = cell_of(p.z, P.minv[q][2], P.cell[q], P.dim[q][2]);
    keys[i] = (uint32_t)(P.base[q] + cx + (long long)P.dim[q][0] * (cy + (long long)P.dim[q][1] * cz));
    least[i] = 0x7fffffff;
}

// The points in sorted order and cell -> its segment s of the sorted order
// (-1 where there are no points).  No segments: the sort gave up, and nothing
// after it may follow its order.
__global__ void gather_kernel(const float4 *__restrict__ pts, const uint32_t *__restrict__ order, int n,
                              const uint32_t *__restrict__ seg_key, const int *__restrict__ nseg,
                              float4 *__restrict__ sorted, int *__restrict__ cell_first) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n || *nseg == 0) return;
    sorted[t] = pts[order[t]];
    if (t < *nseg) cell_first[seg_key[t]] = t;
}

// Union-find over the sorted positions, parent[v] <= v for every v (a root
// links under a smaller one only), so every chain strictly decreases and a
// root is its component's first position.  Reads are volatile (other threads
// link and shorten concurrently); path halving stores a valid ancestor, so any
// interleaving keeps the invariant.
__device__ __forceinline__ int find_root(int *parent, int x) {
    volatile int *p = parent;
    for (int it = 0; it < kUnionLimit; ++it) {
        const int up = p[x];
        if (up == x) return x;
        const int up2 = p[up];
        if (up2 != up) p[x] = up2;
        x = up;
    }
    return -1;
}

// The earlier points that position t has to be tested against: those before it
// in its own cell and in the cell before that, the row of three cells at y - 1
// and the three rows at z - 1 (cells never cross parts; a pair is accepted or
// not whichever of its points comes first).  The cells of a row have
// consecutive keys, so a row's points are one stretch of the sorted order;
// lanes 0..14 of the warp look the 5 x 3 cells up at once.
constexpr int kRows = 5;
struct Rows {
    int from[kRows], to[kRows];  // in ascending order
    float r2;
    __device__ __forceinline__ Rows(int t, uint32_t key, int q, int lane, const int32_t *__restrict__ seg_start, int n,
                                    int nseg, const int *__restrict__ cell_first, const Parts &P) {
        r2 = P.r2[q];
        const unsigned local = key - (uint32_t)P.base[q];
        const unsigned dx0 = P.dim[q][0], dy0 = P.dim[q][1];
        const unsigned row = local / dx0, z0 = row / dy0;
        int first = n, last = 0;
        if (lane < 3 * kRows - 1) {
            const int r = lane / 3;  // (dy, dz) = (-1, -1), (0, -1), (1, -1), (-1, 0), (0, 0)
            const int dx = lane % 3 - 1, dz = r < 3 ? -1 : 0, dy = r < 3 ? r - 1 : r - 4;
            const int x = (int)(local - row * dx0) + dx, y = (int)(row - z0 * dy0) + dy, z = (int)z0 + dz;
            if (x >= 0 && x < (int)dx0 && y >= 0 && y < (int)dy0 && z >= 0) {
                const int s = cell_first[P.base[q] + x + (long long)dx0 * (y + (long long)dy0 * z)];
                if (s >= 0) {
                    first = seg_start[s];
                    last = lane == 3 * kRows - 2 ? t : (s + 1 < nseg ? seg_start[s + 1] : n);
                }
            }
        }
        first = min(first, min(__shfl_down_sync(kAll, first, 1), __shfl_down_sync(kAll, first, 2)));
        last = max(last, max(__shfl_down_sync(kAll, last, 1), __shfl_down_sync(kAll, last, 2)));
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            from[r] = __shfl_sync(kAll, first, 3 * r);
            to[r] = __shfl_sync(kAll, last, 3 * r);
        }
    }
};

__device__ __forceinline__ bool accepted(float4 a, float4 b, float r2) {
    const float ex = __fsub_rn(a.x, b.x), ey = __fsub_rn(a.y, b.y), ez = __fsub_rn(a.z, b.z);
    return __fadd_rn(__fadd_rn(__fmul_rn(ex, ex), __fmul_rn(ey, ey)), __fmul_rn(ez, ez)) <= r2;
}

// First pass, a warp per position t: t hangs under the first earlier point
// that it is joined to.  Nothing but t's warp writes parent[t], and what is left to the
// second pass are the few trees of a component whose roots have no earlier
// neighbour.  With every point its own tree at the start of that pass, all the
// warps of a component contended for the same few roots: 595 us, against 21 for
// this pass, 12 for root_kernel and 91 for what is then left of the second
// (five clouds of 9600 points).  A thread per (point, one of 27 cells, quarter
// of that cell), which tested both orders of every pair and divided 64-bit
// keys for each, took 278 us.
__global__ void __launch_bounds__(kThreads) hook_kernel(
    const float4 *__restrict__ sorted, const uint32_t *__restrict__ keys, int n,
    const int32_t *__restrict__ seg_start, const int *__restrict__ nseg, const int *__restrict__ cell_first,
    const __grid_constant__ Parts P, int *__restrict__ parent) {
    const int t = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (t >= n || *nseg == 0) return;
    const float4 p = sorted[t];
    const Rows R(t, keys[t], __float_as_int(p.w), lane, seg_start, n, *nseg, cell_first, P);
    int up = t;
#pragma unroll
    for (int r = 0; r < kRows; ++r)
        for (int u0 = R.from[r]; u0 < R.to[r] && up == t; u0 += 32) {
            const int u = u0 + lane;
            const unsigned in = __ballot_sync(kAll, u < R.to[r] && accepted(sorted[min(u, n - 1)], p, R.r2));
            if (in) up = u0 + __ffs(in) - 1;
        }
    if (lane == 0) parent[t] = up;
}

__global__ void root_kernel(int *__restrict__ parent, int n, const int *__restrict__ nseg, int *__restrict__ err) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n || *nseg == 0) return;
    const int r = find_root(parent, t);
    if (r < 0) atomicOr(err, 2);
    else parent[t] = r;
}

// Second pass, a warp per position t: the trees of t and of every earlier
// point that it is joined to become one.  A candidate that hangs under t's
// root already costs one read, next to its neighbours'; for the others the warp
// links all roots that it sees under the smallest of them, one atomicCAS each.
// Bound by the latency of its chains (cells, points, parents, roots) at 5 waves
// of warps: its rows read ahead (99 us), rows skipped by their parents before
// the coordinates are read (109 us) and a pass of atomicMin in between (35 us
// for it and 56 for this one) did not help.
__global__ void __launch_bounds__(kThreads) join_kernel(
    const float4 *__restrict__ sorted, const uint32_t *__restrict__ keys, int n,
    const int32_t *__restrict__ seg_start, const int *__restrict__ nseg, const int *__restrict__ cell_first,
    const __grid_constant__ Parts P, int *__restrict__ parent, int *__restrict__ err) {
    const int t = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (t >= n || *nseg == 0) return;
    const float4 p = sorted[t];
    const Rows R(t, keys[t], __float_as_int(p.w), lane, seg_start, n, *nseg, cell_first, P);
    volatile int *up = parent;
    int ri = find_root(parent, t);
    bool bad = ri < 0;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        for (int u0 = R.from[r]; u0 < R.to[r]; u0 += 32) {
            const int u = u0 + lane;
            const float4 c = sorted[min(u, n - 1)];
            int rj = up[min(u, n - 1)];  // of the lanes with an accepted point: a node of its tree, in the end its root
            if (u >= R.to[r] || !accepted(c, p, R.r2)) rj = ri;
            if (rj != ri) rj = find_root(parent, rj);
            for (int it = 0; !__all_sync(kAll, rj == ri); ++it) {
                bad = bad || rj < 0 || it == kUnionLimit;
                if (__any_sync(kAll, bad)) break;
                const int m = min(ri, __reduce_min_sync(kAll, rj));
                if (rj != ri && rj != m) rj = atomicCAS(parent + rj, rj, m) == rj ? m : find_root(parent, rj);
                int rn = ri;
                if (ri != m && lane == 0) rn = atomicCAS(parent + ri, ri, m) == ri ? m : find_root(parent, ri);
                rn = __shfl_sync(kAll, rn, 0);
                if (rj == ri) rj = rn;
                bad = bad || rn < 0;
                ri = rn;
            }
            if (__any_sync(kAll, bad)) {
                if (lane == 0) atomicOr(err, 1);
                return;
            }
        }
    }
}

// The smallest point index of every tree, at its root (least[] starts at INT_MAX).
__global__ void least_kernel(int *__restrict__ parent, const uint32_t *__restrict__ order, int n,
                             const int *__restrict__ nseg, int *__restrict__ least, int *__restrict__ err) {
    if (*nseg == 0) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = t < n ? find_root(parent, t) : -1;
    if (t < n) {
        if (r < 0) atomicOr(err, 2);
        else parent[t] = r;
    }
    const int r0 = __shfl_sync(kAll, r, 0);
    const int i = t < n ? (int)order[t] : 0x7fffffff;
    if (__all_sync(kAll, r == r0 || t >= n)) {  // one tree in the whole warp, as nearly always
        const int m = __reduce_min_sync(kAll, i);
        if ((threadIdx.x & 31) == 0 && r0 >= 0) atomicMin(least + r0, m);
    } else if (r >= 0) {
        atomicMin(least + r, i);
    }
}

// Point index -> label.  The root is looked up again: least_kernel's store of it
// may have been followed by another thread's path halving, whose older ancestor
// is a node of the tree but has no least point.  status[1] collects the errors: a
// sort that gave up is 4.
__global__ void label_kernel(int *__restrict__ parent, const uint32_t *__restrict__ order, int n,
                             const int *__restrict__ nseg, const int *__restrict__ least,
                             const int *__restrict__ sort_err, uint32_t *__restrict__ label,
                             int *__restrict__ status) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0 && *sort_err) atomicOr(status + 1, 4);
    if (t >= n || *nseg == 0) return;
    const int r = find_root(parent, t);
    if (r < 0) atomicOr(status + 1, 2);
    label[order[t]] = r < 0 ? 0u : (uint32_t)least[r];
}

// The clusters of [lo, hi] points, as (first position, points) of the order by
// label; status[0] counts them.
__global__ void cluster_kernel(const int32_t *__restrict__ seg_start, const int *__restrict__ nseg, int n, int lo,
                               int hi, const int *__restrict__ sort_err, int2 *__restrict__ rec,
                               int *__restrict__ status) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s == 0 && *sort_err) atomicOr(status + 1, 4);
    if (s >= *nseg) return;
    const int b = seg_start[s], e = s + 1 < *nseg ? seg_start[s + 1] : n;
    if (e - b >= lo && e - b <= hi) rec[atomicAdd(status, 1)] = make_int2(b, e - b);
}

}  // namespace ec

struct ndt_ec {
    int device = 0;
    cudaStream_t stream = nullptr;
    std::string err;
    void *work = nullptr, *cell_first = nullptr;  // all buffers sized by the points, the cell table
    size_t work_cap = 0, cell_cap = 0;
    char *host = nullptr;  // pinned: the points on their way in, indices and clusters on their way out
    size_t host_cap = 0;
};

namespace {

constexpr long long kMaxCells = 1LL << 28;  // dense cell table (4 B per cell), at most
constexpr int kCopyPoints = 1 << 14;  // points per copy to the device (192 KiB)

int fail(ndt_ec *h, int code, const std::string &msg) {
    if (h) h->err = msg;
    return code;
}

cudaError_t ensure(void **p, size_t *cap, size_t bytes) {
    if (*p && *cap >= bytes) return cudaSuccess;
    if (*p) cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    const size_t want = std::max(bytes + bytes / 2, (size_t)256);
    cudaError_t e = cudaMalloc(p, want);
    if (e == cudaSuccess) *cap = want;
    return e;
}

#define ECK(call)                                                                             \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess) return fail(h, NDT_E_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

// One pass over the points of C.count clouds (C.off[C.count] of them, tolerance[r]
// for ring r).  by_cluster: *index is the point indices, cluster by cluster, and
// rec the clusters of [20, 100000] points in it, by smallest point index;
// otherwise *index is every point's label, the smallest index of its component
// (parts never join).  *points are the handle's copy of the points (the output
// may overlay the input); both are valid until the handle's next call.
constexpr int kMinCluster = 20, kMaxCluster = 100000;

int cluster_pass(ndt_ec *h, const float *xyz, const ec::Clouds &C, const float *tolerance, bool by_cluster,
                 const float **points, const int **index, std::vector<int2> &rec) {
    ndt::NvtxRange range("ec labels");
    rec.clear();
    const int np = C.count * C.rings, N = C.off[C.count];
    if (N == 0) return NDT_OK;
    cudaStream_t st = h->stream;

    // one device and one pinned block, cut into 256-byte aligned pieces
    size_t bytes = 0;
    auto piece = [&bytes](size_t b) {
        const size_t at = bytes;
        bytes += (b + 255) / 256 * 256;
        return at;
    };
    const size_t max_rec = (size_t)N / kMinCluster + 1;
    const size_t o_boxes = piece(sizeof(ec::Box) * ec::kMaxParts), o_status = piece(2 * sizeof(int)),
                 o_rec = piece(sizeof(int2) * max_rec), o_xyz = piece(3 * sizeof(float) * (size_t)N);
    const size_t host_bytes = bytes + sizeof(int) * (size_t)N;  // the indices come last
    const size_t o_pts = piece(sizeof(float4) * (size_t)N), o_sorted = piece(sizeof(float4) * (size_t)N),
                 o_parent = piece(sizeof(int) * (size_t)N), o_least = piece(sizeof(int) * (size_t)N),
                 o_start = piece(sizeof(int) * (size_t)N), o_key = piece(sizeof(int) * (size_t)N),
                 o_sort = piece(ndt::sort_scratch_bytes(N));
    ECK(ensure(&h->work, &h->work_cap, bytes));
    if (h->host_cap < host_bytes) {
        if (h->host) cudaFreeHost(h->host);
        h->host = nullptr;
        h->host_cap = 0;
        ECK(cudaMallocHost((void **)&h->host, host_bytes + host_bytes / 2));
        h->host_cap = host_bytes + host_bytes / 2;
    }
    char *dev = (char *)h->work;
    ec::Box *boxes = (ec::Box *)(dev + o_boxes), *h_boxes = (ec::Box *)(h->host + o_boxes);
    int *status = (int *)(dev + o_status), *err = status + 1, *h_status = (int *)(h->host + o_status);
    int2 *d_rec = (int2 *)(dev + o_rec), *h_rec = (int2 *)(h->host + o_rec);
    float *d_xyz = (float *)(dev + o_xyz), *h_xyz = (float *)(h->host + o_xyz);
    int *h_index = (int *)(h->host + host_bytes - sizeof(int) * (size_t)N);
    float4 *pts = (float4 *)(dev + o_pts), *sorted = (float4 *)(dev + o_sorted);
    int *parent = (int *)(dev + o_parent), *least = (int *)(dev + o_least);
    int32_t *seg_start = (int32_t *)(dev + o_start);
    uint32_t *seg_key = (uint32_t *)(dev + o_key);
    ndt::SortBuffers sb = ndt::sort_buffers(dev + o_sort, N);
    const unsigned blocks = (unsigned)((N + ec::kThreads - 1) / ec::kThreads);

    // parts and boxes; the points go over in pieces, so that the copy into the
    // pinned block runs beside the one to the device
    for (int q = 0; q < np; ++q)
        h_boxes[q] = {{INT_MAX, INT_MAX, INT_MAX}, {INT_MIN, INT_MIN, INT_MIN}, 0, 0};
    h_status[0] = h_status[1] = 0;
    ECK(cudaMemcpyAsync(boxes, h_boxes, o_status + 2 * sizeof(int) - o_boxes, cudaMemcpyHostToDevice, st));
    for (int i = 0; i < N; i += kCopyPoints) {
        const size_t at = 3 * (size_t)i, len = 3 * sizeof(float) * (size_t)std::min(kCopyPoints, N - i);
        std::memcpy(h_xyz + at, xyz + at, len);
        ECK(cudaMemcpyAsync(d_xyz + at, h_xyz + at, len, cudaMemcpyHostToDevice, st));
    }
    ec::part_kernel<<<blocks, ec::kThreads, 0, st>>>(d_xyz, N, C, pts, boxes);
    ECK(cudaGetLastError());
    ECK(cudaMemcpyAsync(h_boxes, boxes, sizeof(ec::Box) * np, cudaMemcpyDeviceToHost, st));
    ECK(cudaStreamSynchronize(st));

    ec::Parts P;
    std::memset(&P, 0, sizeof(P));
    long long cells = 0;
    for (int q = 0; q < np; ++q) {
        const ec::Box &b = h_boxes[q];
        const float tol = tolerance[q % C.rings];
        P.base[q] = cells;
        P.cell[q] = tol * 1.0001f;  // cells a little wider than the radius
        P.r2[q] = tol * tol;
        if (!b.points) continue;
        if (b.bad) return fail(h, NDT_E_ARG, "non-finite point coordinates");
        long long G = 1;
        for (int k = 0; k < 3; ++k) {
            const int lo = ec::ordered(b.lo[k]), hi = ec::ordered(b.hi[k]);
            float mn, mx;
            std::memcpy(&mn, &lo, sizeof(mn));
            std::memcpy(&mx, &hi, sizeof(mx));
            P.minv[q][k] = mn;
            const double d = std::floor(((double)mx - (double)mn) / (double)P.cell[q]) + 1.0;
            if (!(d >= 1.0 && d < 2147483647.0)) return fail(h, NDT_E_CAPACITY, "a cloud spans too many cells");
            P.dim[q][k] = (int)d;
            G *= P.dim[q][k];
            if (G > kMaxCells) break;
        }
        cells += G;
        if (cells > kMaxCells) return fail(h, NDT_E_CAPACITY, "the clouds span more than 2^28 cells of the tolerance");
    }
    P.base[np] = cells;
    auto bits_for = [](long long values) {
        int bits = 1;
        while (bits < 31 && (1LL << bits) < values) ++bits;
        return bits;
    };
    ECK(ensure(&h->cell_first, &h->cell_cap, sizeof(int) * (size_t)cells));
    int *cell_first = (int *)h->cell_first;
    ECK(cudaMemsetAsync(cell_first, 0xff, sizeof(int) * (size_t)cells, st));
    ec::key_kernel<<<blocks, ec::kThreads, 0, st>>>(pts, N, P, sb.k0, least);
    ndt::sort_segments(sb, N, bits_for(cells), seg_start, seg_key, st, true);
    ec::gather_kernel<<<blocks, ec::kThreads, 0, st>>>(pts, sb.v0, N, seg_key, sb.nseg, sorted, cell_first);
    const unsigned per_block = ec::kThreads / 32, wide = (N + per_block - 1) / per_block;
    ec::hook_kernel<<<wide, ec::kThreads, 0, st>>>(sorted, sb.k0, N, seg_start, sb.nseg, cell_first, P, parent);
    ec::root_kernel<<<blocks, ec::kThreads, 0, st>>>(parent, N, sb.nseg, err);
    ec::join_kernel<<<wide, ec::kThreads, 0, st>>>(sorted, sb.k0, N, seg_start, sb.nseg, cell_first, P, parent, err);
    ec::least_kernel<<<blocks, ec::kThreads, 0, st>>>(parent, sb.v0, N, sb.nseg, least, err);
    ec::label_kernel<<<blocks, ec::kThreads, 0, st>>>(parent, sb.v0, N, sb.nseg, least, ndt::sort_error(sb, N), sb.k0,
                                                      status);
    if (by_cluster) {
        ndt::sort_segments(sb, N, bits_for(N), seg_start, seg_key, st, true);
        ec::cluster_kernel<<<blocks, ec::kThreads, 0, st>>>(seg_start, sb.nseg, N, kMinCluster, kMaxCluster,
                                                            ndt::sort_error(sb, N), d_rec, status);
    }
    ECK(cudaGetLastError());
    ECK(cudaMemcpyAsync(h_status, status, by_cluster ? o_rec + sizeof(int2) * max_rec - o_status : 2 * sizeof(int),
                        cudaMemcpyDeviceToHost, st));
    ECK(cudaMemcpyAsync(h_index, by_cluster ? sb.v0 : sb.k0, sizeof(int) * (size_t)N, cudaMemcpyDeviceToHost, st));
    ECK(cudaStreamSynchronize(st));
    if (h_status[1] & 4) return fail(h, NDT_E_CUDA, "a wait between the sort's tiles gave up");
    if (h_status[1]) return fail(h, NDT_E_CUDA, "union-find retry limit reached");
    *points = h_xyz;
    *index = h_index;
    if (by_cluster) {
        rec.assign(h_rec, h_rec + h_status[0]);
        std::sort(rec.begin(), rec.end(), [](int2 a, int2 b) { return a.x < b.x; });
    }
    return NDT_OK;
}

// Labels of one cloud.
int labels_of(ndt_ec *h, const float *xyz, int n, float tolerance, const int **labels) {
    ec::Clouds C;
    std::memset(&C, 0, sizeof(C));
    C.count = C.rings = 1;
    C.off[1] = n;
    const float *points;
    std::vector<int2> none;
    return cluster_pass(h, xyz, C, &tolerance, false, &points, labels, none);
}

// The reference's clusters from component labels: components in order of
// their smallest index, indices ascending, sizes in [lo, hi], then ordered by
// size with std::sort over reverse iterators (extract, kernel.cpp:635-647).
void clusters_of(const int *labels, int n, int lo, int hi, std::vector<std::vector<int>> &out) {
    std::vector<int> size(n, 0), slot(n, -1);
    for (int i = 0; i < n; ++i) ++size[labels[i]];
    out.clear();
    for (int i = 0; i < n; ++i)
        if (labels[i] == i && size[i] >= lo && size[i] <= hi) {
            slot[i] = (int)out.size();
            out.emplace_back();
            out.back().reserve(size[i]);
        }
    for (int i = 0; i < n; ++i)
        if (slot[labels[i]] >= 0) out[slot[labels[i]]].push_back(i);
    std::sort(out.rbegin(), out.rend(),
              [](const std::vector<int> &a, const std::vector<int> &b) { return a.size() < b.size(); });
}

}  // namespace

extern "C" {

int ndt_ec_create(int device, ndt_ec **out) {
    if (!out) return NDT_E_ARG;
    *out = nullptr;
    ndt_ec *h = new ndt_ec();
    h->device = device;
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = (cudaError_t)ndt::prepare_sort();
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        delete h;
        return NDT_E_CUDA;
    }
    *out = h;
    return NDT_OK;
}

void ndt_ec_destroy(ndt_ec *h) {
    if (!h) return;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    for (void *p : {h->work, h->cell_first})
        if (p) cudaFree(p);
    if (h->host) cudaFreeHost(h->host);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
}

const char *ndt_ec_last_error(const ndt_ec *h) { return h ? h->err.c_str() : "null handle"; }

int ndt_ec_labels(ndt_ec *h, const float *xyz, int n, float tolerance, int *labels) {
    if (!h || n < 0 || (n > 0 && (!xyz || !labels)) || !(tolerance > 0.0f) || !std::isfinite(tolerance))
        return fail(h, NDT_E_ARG, "bad argument");
    ECK(cudaSetDevice(h->device));
    const int *lab = nullptr;
    if (int rc = labels_of(h, xyz, n, tolerance, &lab)) return rc;
    if (n) std::memcpy(labels, lab, sizeof(int) * (size_t)n);
    return NDT_OK;
}

int ndt_ec_extract(ndt_ec *h, const float *xyz, int n, float tolerance, int min_size, int max_size,
                   int *num_clusters, int *cluster_offsets, int *cluster_indices) {
    if (!h || n < 0 || (n > 0 && !xyz) || !num_clusters || !cluster_offsets || !cluster_indices ||
        !(tolerance > 0.0f) || !std::isfinite(tolerance))
        return fail(h, NDT_E_ARG, "bad argument");
    ECK(cudaSetDevice(h->device));
    const int *lab = nullptr;
    if (int rc = labels_of(h, xyz, n, tolerance, &lab)) return rc;
    std::vector<std::vector<int>> cl;
    clusters_of(lab, n, min_size, max_size, cl);
    int pos = 0;
    cluster_offsets[0] = 0;
    for (size_t c = 0; c < cl.size(); ++c) {
        std::memcpy(cluster_indices + pos, cl[c].data(), sizeof(int) * cl[c].size());
        pos += (int)cl[c].size();
        cluster_offsets[c + 1] = pos;
    }
    *num_clusters = (int)cl.size();
    return NDT_OK;
}

// segmentByDistance (kernel.cpp:767-814) with clusterAndColor (:652-765):
// five rings of distance from the sensor (< 15, 30, 45, 60 m, beyond) with
// tolerances 0.5, 1.1, 1.6, 2.3 and 2.6f, clusters of 20 to 100000 points.
// Clouds [c0, c1) of a packed batch in one GPU pass; outputs appended at the
// running counts np / nb.
namespace {
int segment_clouds(ndt_ec *h, const float *xyz, const int *offsets, int c0, int c1, float *out_xyz, int *out_off,
                   double *boxes, int *box_off, double *centroids, int &np, int &nb) {
    const float tol[ec::kRings] = {0.5f, 1.1f, 1.6f, 2.3f, 2.6f};
    ec::Clouds C;
    std::memset(&C, 0, sizeof(C));
    C.count = c1 - c0;
    C.rings = ec::kRings;
    for (int c = 0; c <= C.count; ++c) C.off[c] = offsets[c0 + c] - offsets[c0];
    const float *points = nullptr;
    const int *index = nullptr;
    std::vector<int2> rec;  // every ring of every cloud in one pass
    if (int rc = cluster_pass(h, xyz + 3 * (size_t)offsets[c0], C, tol, true, &points, &index, rec)) return rc;
    // by part, in order of the smallest index, then by size as extract() orders them
    std::vector<std::vector<int2>> part((size_t)C.count * ec::kRings);
    for (int2 r : rec) {
        const int i = index[r.x];
        const float *q = points + 3 * (size_t)i;
        part[(size_t)ec::kRings * ec::cloud_of(C, i) + ec::ring_of(q[0], q[1])].push_back(r);
    }
    std::vector<ec::ClusterJob> jobs;
    jobs.reserve(rec.size());
    std::vector<size_t> first(C.count + 1, 0);  // each cloud's first cluster
    for (int c = 0; c < C.count; ++c) {
        out_off[c0 + c] = np;
        for (int r = 0; r < ec::kRings; ++r) {
            std::vector<int2> &cl = part[(size_t)ec::kRings * c + r];
            std::sort(cl.rbegin(), cl.rend(), [](const int2 &a, const int2 &b) { return a.y < b.y; });
            for (int2 k : cl) {
                jobs.push_back({index + k.x, k.y, out_xyz + 3 * (size_t)np});
                np += k.y;
            }
        }
        first[c + 1] = jobs.size();
    }
    out_off[c1] = np;
    {
        ndt::NvtxRange range("ec boxes");
        ec::finish_clusters(points, jobs.data(), (int)jobs.size());
    }
    for (int c = 0; c < C.count; ++c) {
        box_off[c0 + c] = nb;
        for (size_t j = first[c]; j < first[c + 1]; ++j) {
            if (!jobs[j].kept) continue;
            std::memcpy(boxes + 10 * (size_t)nb, jobs[j].box, sizeof(jobs[j].box));
            std::memcpy(centroids + 3 * (size_t)nb, jobs[j].centroid, sizeof(jobs[j].centroid));
            ++nb;
        }
    }
    box_off[c1] = nb;
    return NDT_OK;
}
}  // namespace

int ndt_ec_segment(ndt_ec *h, const float *xyz, int n, float *out_xyz, int *out_n, double *boxes, int *num_boxes,
                   double *centroids, int *num_centroids) {
    if (!h || n < 0 || (n > 0 && !xyz) || !out_xyz || !out_n || !boxes || !num_boxes || !centroids ||
        !num_centroids)
        return fail(h, NDT_E_ARG, "bad argument");
    ECK(cudaSetDevice(h->device));
    const int off[2] = {0, n};
    int oo[2], bo[2], np = 0, nb = 0;
    if (int rc = segment_clouds(h, xyz, off, 0, 1, out_xyz, oo, boxes, bo, centroids, np, nb)) return rc;
    *out_n = np;
    *num_boxes = nb;
    *num_centroids = nb;
    return NDT_OK;
}

int ndt_ec_box_yaw(const float *xyz, int n, double *qz, double *qw) {
    if (n < 0 || (n > 0 && !xyz) || !qz || !qw) return NDT_E_ARG;
    float lo[2] = {std::numeric_limits<float>::max(), std::numeric_limits<float>::max()};
    for (int i = 0; i < n; ++i)
        for (int k = 0; k < 2; ++k) {
            const float v = xyz[3 * (size_t)i + k];
            if (!std::isfinite(v)) return NDT_E_ARG;
            if (v < lo[k]) lo[k] = v;
        }
    ec::box_yaw(xyz, n, lo[0], lo[1], qz, qw);
    return NDT_OK;
}

int ndt_ec_box_yaws(int C, const float *xyz, const int *offsets, double *qz, double *qw) {
    if (C < 0 || (C > 0 && (!offsets || !qz || !qw)) || (C > 0 && offsets[0] != 0)) return NDT_E_ARG;
    if (C > 0 && offsets[C] > 0 && !xyz) return NDT_E_ARG;
    std::vector<ec::YawJob> jobs(C);
    for (int c = 0; c < C; ++c) {
        if (offsets[c + 1] < offsets[c]) return NDT_E_ARG;
        float lo[2] = {std::numeric_limits<float>::max(), std::numeric_limits<float>::max()};
        for (int i = offsets[c]; i < offsets[c + 1]; ++i)
            for (int k = 0; k < 2; ++k) {
                const float v = xyz[3 * (size_t)i + k];
                if (!std::isfinite(v)) return NDT_E_ARG;
                if (v < lo[k]) lo[k] = v;
            }
        jobs[c] = {xyz + 3 * (size_t)offsets[c], offsets[c + 1] - offsets[c], lo[0], lo[1], qz + c, qw + c};
    }
    ec::box_yaws(jobs.data(), C);
    return NDT_OK;
}

int ndt_ec_segment_batch(ndt_ec *h, int C, const float *xyz, const int *offsets, float *out_xyz, int *out_offsets,
                         double *boxes, int *box_offsets, double *centroids) {
    if (!h || C <= 0 || !offsets || !out_xyz || !out_offsets || !boxes || !box_offsets || !centroids ||
        (offsets[C] > 0 && !xyz) || offsets[0] != 0)
        return fail(h, NDT_E_ARG, "bad argument");
    for (int c = 0; c < C; ++c)
        if (offsets[c + 1] < offsets[c]) return fail(h, NDT_E_ARG, "offsets must be non-decreasing");
    ECK(cudaSetDevice(h->device));
    int np = 0, nb = 0;
    const int per_pass = ec::kMaxParts / 5;
    for (int c0 = 0; c0 < C; c0 += per_pass) {
        const int c1 = std::min(C, c0 + per_pass);
        if (int rc = segment_clouds(h, xyz, offsets, c0, c1, out_xyz, out_offsets, boxes, box_offsets, centroids,
                                    np, nb))
            return rc;
    }
    return NDT_OK;
}

}  // extern "C"
