// Scan pre-filter: voxel-grid downsampling of a batch of raw scans on the
// device (the step that produces the align call's "filtered scan" upstream;
// it is not part of the reference kernel).
//
// Semantics (pinned by oracle/voxel_filter_ref.py):
//   * a point is kept when x, y, z are finite;
//   * its leaf is (floor(x * r), floor(y * r), floor(z * r)) with
//     r = 1 / leaf rounded to float and each product rounded to float (the
//     leaf index of the point-cloud library's voxel-grid filter, which
//     Autoware's mapping pipeline runs with a 2 m leaf before the align);
//   * every occupied leaf of a scan yields one point: the mean of its points,
//     summed in FP64 in input order and divided by their count, rounded to
//     float (x, y, z and the fourth component alike);
//   * a scan's output points are ordered by leaf, x fastest, then y, then z.
//
// Device pipeline for B scans: the leaf bounding box of every scan (warps
// over the packed points, 64-bit atomics) and its leaf-key range, then one of
//   * scan_kernel, when every scan's points and leaves fit a block's shared
//     memory (scan_fits): one block per scan does it all;
//   * the general path: an exclusive scan of the ranges gives every scan a
//     disjoint key interval, so one 32-bit key per point (scan interval base +
//     local leaf key) orders points by scan, then leaf; one stable radix sort
//     and segmentation of all points (shared with the voxel-grid build); the
//     points gathered into key order; per segment the FP64 mean in input
//     order; output offsets by lower bounds of the scans' key bases in the
//     sorted segment keys.
#include <cuda_runtime.h>
#include <stdint.h>

#include <climits>
#include <cmath>
#include <cstring>
#include <string>

#include "../../include/ndt_b200.h"
#include "chain.cuh"
#include "grid_build.h"
#include "nvtx_range.h"

namespace vf {

constexpr int kThreads = 256;

__device__ __forceinline__ bool finite3(float4 p) { return isfinite(p.x) && isfinite(p.y) && isfinite(p.z); }

// The product is clamped to +-2^60 before the integer conversion, so that
// any finite coordinate has a defined leaf index (a scan that far out fails
// the 2^31-leaf range check).
__device__ __forceinline__ long long leaf_of(float v, float r) {
    float q = floorf(__fmul_rn(v, r));
    q = fminf(fmaxf(q, -1.1529215e18f), 1.1529215e18f);  // 2^60
    return (long long)q;
}

struct ScanGeom {
    long long lo[3];  // leaf index minimum per axis
    long long d[3];   // leaf extent per axis
};

// Scan of point (or key) i: the last b in [0, B) with first[b] <= i, for a
// non-decreasing first[] (point offsets, or key bases: with empty scans the
// search lands on the scan that owns i).
__device__ __forceinline__ int owner(const int *__restrict__ first, int B, int i) {
    int lo = 0, hi = B;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(first + mid) <= i) lo = mid; else hi = mid;
    }
    return lo;
}

constexpr int kBoxWarpPoints = 1024;  // points per warp in the box pass

// Leaf bounding boxes: box[6 b .. 6 b + 5] = min x, y, z, max x, y, z leaf
// index of scan b's finite points, by 64-bit atomics (order-independent).
// Each warp walks kBoxWarpPoints consecutive points, 4 steps of 32 at a time,
// and keeps a per-lane box of the coordinates (the leaf index does not
// decrease with the coordinate, so the box's corners give the leaf box) while
// the points stay in one scan; steps that cross a scan boundary flush it and
// settle their points one by one.  Bound by the read of the points: 16.7M
// points 79 -> 45 us against boxes of 64-bit leaf indices, one step at a time.
__device__ __forceinline__ void box_flush(long long *__restrict__ box, int b, float r, float (&mn)[3], float (&mx)[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mn[k] = fminf(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
            mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
        }
    if ((threadIdx.x & 31) == 0 && mn[0] <= mx[0])
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            atomicMin(box + 6 * b + k, leaf_of(mn[k], r));
            atomicMax(box + 6 * b + 3 + k, leaf_of(mx[k], r));
        }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        mn[k] = INFINITY;
        mx[k] = -INFINITY;
    }
}

__global__ void box_kernel(const float4 *__restrict__ pts, const int *__restrict__ offsets, int B, int n, float r,
                           long long *__restrict__ box) {
    constexpr int kSteps = 4;
    const int lane = threadIdx.x & 31;
    const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long w0l = gw * kBoxWarpPoints;
    if (w0l >= n) return;
    const int w0 = (int)w0l, w1 = n - w0 < kBoxWarpPoints ? n : w0 + kBoxWarpPoints;
    int cur = owner(offsets, B, w0);
    int hi = __ldg(offsets + cur + 1);
    float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    auto take = [&](float4 p) {
        if (!finite3(p)) return;
        mn[0] = fminf(mn[0], p.x); mn[1] = fminf(mn[1], p.y); mn[2] = fminf(mn[2], p.z);
        mx[0] = fmaxf(mx[0], p.x); mx[1] = fmaxf(mx[1], p.y); mx[2] = fmaxf(mx[2], p.z);
    };
    for (int base = w0; base < w1; base += 32 * kSteps) {
        const int last = w1 - base < 32 * kSteps ? w1 - 1 : base + 32 * kSteps - 1;
        if (last < hi) {  // warp-uniform: all of the steps' points lie in scan cur
            float4 p[kSteps];
#pragma unroll
            for (int k = 0; k < kSteps; ++k) p[k] = pts[min(base + 32 * k + lane, last)];
#pragma unroll
            for (int k = 0; k < kSteps; ++k) take(p[k]);  // (a point taken twice changes no box)
            continue;
        }
        box_flush(box, cur, r, mn, mx);
        for (int i = base + lane; i <= last; i += 32) {
            const float4 p = pts[i];
            if (!finite3(p)) continue;
            const int b = owner(offsets, B, i);
            const float v[3] = {p.x, p.y, p.z};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const long long q = leaf_of(v[k], r);
                atomicMin(box + 6 * b + k, q);
                atomicMax(box + 6 * b + 3 + k, q);
            }
        }
        if (last + 1 < w1) {
            cur = owner(offsets, B, last + 1);
            hi = __ldg(offsets + cur + 1);
        }
    }
    box_flush(box, cur, r, mn, mx);
}

__global__ void box_init_kernel(long long *__restrict__ box, int B) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 6 * B; i += gridDim.x * blockDim.x)
        box[i] = (i % 6) < 3 ? LLONG_MAX : LLONG_MIN;
}

// One block: per scan its geometry and key range (dx * dy * dz, 0 without
// finite points), the exclusive scan of the ranges into key bases
// (base[B] = total), and the box reset for the next call.  flags[0] |= 1 when
// a scan spans 2^31 leaves or more, |= 2 when the batch spans 2^31 - 1 or
// more; flags[1] = total; flags[2], flags[3] = the largest leaf range and point
// count of a scan (INT_MAX when the offsets are not a partition of the n points
// into scans: the boxes then hold each point in one scan, as the general path
// takes them, and the ranges of points say something else).
constexpr int kRangeThreads = 1024;

__global__ void __launch_bounds__(kRangeThreads) range_kernel(long long *__restrict__ box, int B,
                                                              const int *__restrict__ offsets, int n,
                                                              ScanGeom *__restrict__ geom, int *__restrict__ base,
                                                              int *__restrict__ flags) {
    __shared__ long long s_sum[kRangeThreads];
    const int t = threadIdx.x;
    if (t == 0 && (offsets[0] != 0 || offsets[B] != n)) atomicMax(flags + 3, INT_MAX);
    const int per = (B + kRangeThreads - 1) / kRangeThreads;
    const int b0 = t * per, b1 = b0 + per < B ? b0 + per : B;
    long long local = 0;
    int err = 0;
    for (int b = b0; b < b1; ++b) {
        ScanGeom g;
        long long span = 0;
        const long long *bx = box + 6 * b;
        if (bx[0] <= bx[3]) {
            span = 1;
            for (int k = 0; k < 3; ++k) {
                g.lo[k] = bx[k];
                g.d[k] = bx[3 + k] - bx[k] + 1;
                span = (span > (1LL << 31) / g.d[k]) ? (1LL << 32) : span * g.d[k];
            }
        } else {
            for (int k = 0; k < 3; ++k) {
                g.lo[k] = 0;
                g.d[k] = 1;
            }
        }
        if (span >= (1LL << 31)) {
            err |= 1;
            span = 0;
        }
        atomicMax(flags + 2, (int)span);
        // (+ 1: a leaf that may hold all of a scan's points, which scan_kernel's 16-bit counts must not)
        const int o0 = offsets[b], o1 = offsets[b + 1];
        atomicMax(flags + 3, o0 >= 0 && o0 <= o1 && o1 <= n ? o1 - o0 + (span <= 1 ? 1 : 0) : INT_MAX);
        geom[b] = g;
        base[b] = (int)span;  // the range for now; the scan below makes it a base
        local += span;
        for (int k = 0; k < 6; ++k) box[6 * b + k] = k < 3 ? LLONG_MAX : LLONG_MIN;
    }
    s_sum[t] = local;
    __syncthreads();
    for (int o = 1; o < kRangeThreads; o <<= 1) {  // inclusive Hillis-Steele scan
        const long long v = t >= o ? s_sum[t - o] : 0;
        __syncthreads();
        s_sum[t] += v;
        __syncthreads();
    }
    long long run = s_sum[t] - local;
    const long long total = s_sum[kRangeThreads - 1];
    const long long cap = 0x7fffffffLL;
    for (int b = b0; b < b1; ++b) {
        const int span = base[b];
        base[b] = (int)(run < cap ? run : cap);
        run += span;
    }
    if (err) atomicOr(flags, 1);
    if (t == 0) {
        if (total >= cap) atomicOr(flags, 2);
        base[B] = (int)(total < cap ? total : cap);
        flags[1] = (int)(total < cap ? total : cap);
    }
}

// ---------------------------------------------------------------------------
// One block per scan: the leaves' point counts in shared memory (16 bits
// each), their prefix sums, the points' indices scattered to their leaves
// (atomics: in any order within a leaf), the list of occupied leaves, and the
// means.  A leaf's points are added in any order when that is exact (see
// Magnitudes), so that the result is the in-order sum bit for bit; otherwise in
// input order.  A leaf of at most kGroupLeaf points is 4 lanes' (a thread per
// leaf waits for its warp's largest leaf: means of 256 scans 205 -> 180 us),
// whose first sorts the indices in the latter case; a larger one is a warp's
// (which sorts them too, or, beyond kSortLeaf points, walks the scan's keys in
// order).
// The output's place comes from the occupied leaves of the scans before,
// chained over the blocks.  The points are read twice, the second time in leaf
// order, and the leaf keys written and read once in between.  The call on 256 scans of 65536
// points with 2 m leaves: 1081 us on the general path, 379 us with this kernel
// (276 us of it, bound by the gathers and the instructions of the means: counts
// 60, prefixes 10, scatter 24, means 180).
constexpr int kScanThreads = 1024, kScanWarps = kScanThreads / 32;
constexpr int kGroupLeaf = 64;
constexpr int kSortLeaf = 2048;
constexpr int kScanMaxPoints = 65536;             // indices within a scan in 16 bits
constexpr int kScanMaxLeaves = 65535;             // leaf keys in 16 bits, one value for dropped points
constexpr size_t kScanSmem = 220 * 1024;

__host__ __device__ inline size_t scan_words(int leaves) { return ((size_t)leaves + 3) / 2; }  // 2 counts per word

// Shared memory of a scan of n points and `leaves` leaves: counts, occupied
// leaves, indices.
__host__ __device__ inline size_t scan_smem(int leaves, int n) {
    const size_t list = leaves < n ? (size_t)leaves : (size_t)n;
    return 4 * scan_words(leaves) + 4 * ((list + 1) / 2) + 2 * (size_t)n + 16;
}

inline bool scan_fits(int leaves, int n) {
    return n <= kScanMaxPoints && leaves <= kScanMaxLeaves && scan_smem(leaves, n) <= kScanSmem;
}

// Whether it also pays.  A block's time goes with its scan, the general path's
// with the batch, spread over the chip: calls of about 77 us + 1.17 ns per
// point of the longest scan against 100 us + 0.065 ns per point of the batch
// (65536 points a scan, 1 / 8 / 12 / 20 / 40 scans: 146 / 153 / 154 / 156 /
// 154 us against 111 / 134 / 150 / 185 / 250; 1 / 8 scans of 30000 points: 113
// / 119 against 103 / 129; one of 2000: 80 against 96).
inline bool scan_pays(int longest, int total) { return longest <= 20000 + total / 18; }

// Whether a_bytes at a and b_bytes at b share any.  scan_kernel writes a scan's results
// while other blocks still read theirs, so outputs over inputs (an in-place
// call) take the general path, which has read all before it writes.
inline bool overlap(const void *a, size_t a_bytes, const void *b, size_t b_bytes) {
    const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b;
    return x < y + b_bytes && y < x + a_bytes;
}

struct ScanArgs {
    const float4 *pts;
    const int *offsets;
    const ScanGeom *geom;
    float r;
    int B;
    int leaves, n;    // the largest of any scan (the layout of shared memory)
    uint16_t *keys;   // scratch: one per point
    float4 *out;
    int *out_off;
    int *ticket;      // zero on entry
    uint64_t *state;  // B chained counts, zero on entry
    int *err;         // set when a wait gave up
};

// Local leaf key of a finite point, or -1.  (Every finite point of the scan
// lies in its box, whose extents fit 32 bits; `small`: its corners do, too.)
struct LocalGrid {
    long long lo[3];
    int d[3];
    float r;
    bool small;
    __device__ __forceinline__ int axis(float v, int k) const {
        return small ? (int)floorf(__fmul_rn(v, r)) - (int)lo[k] : (int)(leaf_of(v, r) - lo[k]);
    }
    __device__ __forceinline__ int key(float4 p) const {
        if (!finite3(p)) return -1;
        return axis(p.x, 0) + d[0] * (axis(p.y, 1) + d[1] * axis(p.z, 2));
    }
};

// Sums of floats in FP64 are exact, in any order, when every partial sum is a
// multiple of the smallest value's last bit and below 2^53 of them: with
// exponents in [lo, hi], 24-bit significands and m values, when
// hi - lo + 24 + ceil(log2 m) <= 53.  Zeros count for nothing; infinities and
// NaN never pass.  lo and hi hold magnitudes' bits, lo less one (a zero's wraps
// to the largest).
struct Magnitudes {
    unsigned lo = 0xffffffffu, hi = 0u;
    __device__ __forceinline__ void take(float v) {
        const unsigned u = __float_as_uint(v) & 0x7fffffffu;
        hi = max(hi, u);
        lo = min(lo, u - 1u);
    }
    __device__ __forceinline__ bool exact(int m) const {
        if (hi >= 0x7f800000u) return false;
        if (hi == 0u) return true;
        const int l = max(1, (int)((lo + 1u) >> 23)), h = max(1, (int)(hi >> 23));  // subnormals: exponent 1's last bit
        return h - l + 24 + (m > 1 ? 32 - __clz(m - 1) : 0) <= 53;
    }
};

__device__ __forceinline__ float4 mean_of(double sx, double sy, double sz, double sw, int m) {
    const double c = (double)m;
    return make_float4((float)(sx / c), (float)(sy / c), (float)(sz / c), (float)(sw / c));
}

// Ascending sort of m indices in shared memory by one warp: the bitonic
// network whose steps all compare upwards (each merge begins with a mirrored
// step), positions beyond m standing for the largest value.
__device__ __forceinline__ void warp_sort(uint16_t *x, int m) {
    const int lane = threadIdx.x & 31;
    for (int size = 2; size < 2 * m; size <<= 1)
        for (int step = size >> 1; step > 0; step >>= 1) {
            __syncwarp();
            for (int c = lane; c < (m + 1) / 2 + step; c += 32) {
                const int i = 2 * step * (c / step) + c % step;  // the lower of the pair
                const int j = step == size >> 1 ? (i | (size - 1)) - (i & (size - 1)) : i + step;
                if (j < m) {
                    const uint16_t a = x[i], b = x[j];
                    if (a > b) {
                        x[i] = b;
                        x[j] = a;
                    }
                }
            }
        }
    __syncwarp();
}

__global__ void __launch_bounds__(kScanThreads) scan_kernel(const __grid_constant__ ScanArgs a) {
    constexpr unsigned kAll = 0xffffffffu;
    extern __shared__ __align__(16) unsigned char s_dyn[];
    unsigned *s_cnt = reinterpret_cast<unsigned *>(s_dyn);  // two 16-bit leaf counters per word
    uint16_t *s_end = reinterpret_cast<uint16_t *>(s_dyn);
    const int list_cap = a.leaves < a.n ? a.leaves : a.n;
    uint16_t *s_list = reinterpret_cast<uint16_t *>(s_cnt + scan_words(a.leaves));
    uint16_t *s_idx = s_list + 2 * ((list_cap + 1) / 2);
    __shared__ unsigned s_warp[2][kScanWarps];
    __shared__ int s_scan, s_wrap, s_base, s_big;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    if (t == 0) {
        s_scan = atomicAdd(a.ticket, 1);
        s_wrap = 0x7fffffff;
        s_big = 0;
    }
    __syncthreads();
    const int b = s_scan;
    const ScanGeom g = a.geom[b];
    LocalGrid G;
    G.r = a.r;
    G.small = true;
    for (int k = 0; k < 3; ++k) {
        G.lo[k] = g.lo[k];
        G.d[k] = (int)g.d[k];
        if (g.lo[k] < -(1LL << 30) || g.lo[k] + g.d[k] > (1LL << 30)) G.small = false;
    }
    const int S = G.d[0] * G.d[1] * G.d[2];
    const int start = a.offsets[b], n = a.offsets[b + 1] - start;
    const float4 *pts = a.pts + start;
    uint16_t *keys = a.keys + start;
    for (int k = t; k < (int)scan_words(S); k += kScanThreads) s_cnt[k] = 0;
    __syncthreads();
    // 1. counts
    for (int i0 = 0; i0 < n; i0 += 4 * kScanThreads) {
        float4 p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = i0 + u * kScanThreads + t;
            if (i < n) p[u] = pts[i];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i0 + u * kScanThreads + t < n) {
                const int k = G.key(p[u]);
                keys[i0 + u * kScanThreads + t] = (uint16_t)k;  // (-1: 0xffff)
                if (k >= 0) atomicAdd(s_cnt + (k >> 1), 1u << (16 * (k & 1)));
            }
    }
    __syncthreads();
    // 2. exclusive prefixes in place, and the occupied leaves in order: each
    // thread takes a run of words
    const int words = (S + 1) / 2, per = (words + kScanThreads - 1) / kScanThreads;
    const int k0 = min(words, t * per), k1 = min(words, k0 + per);
    unsigned sum = 0, occ = 0;
    for (int k = k0; k < k1; ++k) {
        const unsigned c = s_cnt[k];
        sum += (c & 0xffffu) + (c >> 16);
        occ += ((c & 0xffffu) != 0u) + ((c >> 16) != 0u);
    }
    unsigned is = sum, io = occ;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned x = __shfl_up_sync(kAll, is, o), y = __shfl_up_sync(kAll, io, o);
        if (lane >= o) {
            is += x;
            io += y;
        }
    }
    if (lane == 31) {
        s_warp[0][w] = is;
        s_warp[1][w] = io;
    }
    __syncthreads();
    unsigned before = 0, rank = 0, total = 0;
    for (int k = 0; k < kScanWarps; ++k) {
        if (k < w) {
            before += s_warp[0][k];
            rank += s_warp[1][k];
        }
        total += s_warp[1][k];
    }
    before += is - sum;
    rank += io - occ;
    for (int k = k0; k < k1; ++k) {
        const unsigned c = s_cnt[k], c0 = c & 0xffffu, c1 = c >> 16;
        if (c0) s_list[rank++] = (uint16_t)(2 * k);
        if (c1) s_list[rank++] = (uint16_t)(2 * k + 1);
        s_cnt[k] = (before & 0xffffu) | ((before + c0) << 16);
        // (a scan of 2^16 points: the end of its last leaf does not fit 16 bits)
        if (c0 && before + c0 == 65536u) s_wrap = 2 * k;
        if (c1 && before + c0 + c1 == 65536u) s_wrap = 2 * k + 1;
        before += c0 + c1;
    }
    // the scan's place in the output
    if (w == 0) {
        bool bad = false;
        if (lane == 0) ndt::Chain<uint64_t>::publish(a.state + b, b == 0 ? ndt::kUpToSum : ndt::kOwnSum, total);
        const uint64_t base = ndt::warp_chain_before(a.state, b, bad);
        if (lane == 0) {
            if (bad)
                atomicOr(a.err, 1);
            else
                ndt::Chain<uint64_t>::publish(a.state + b, ndt::kUpToSum, base + total);
            s_base = bad ? -1 : (int)base;
            a.out_off[b] = (int)base;
            if (b == a.B - 1) a.out_off[a.B] = (int)(base + total);
        }
    }
    __syncthreads();
    if (s_base < 0) return;
    // 3. indices to their leaves: afterwards s_end[k] is the end of leaf k's run
    // (each thread reads back the keys it wrote)
    for (int i0 = 0; i0 < n; i0 += 8 * kScanThreads) {
        unsigned k[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int i = i0 + u * kScanThreads + t;
            k[u] = i < n ? keys[i] : 0xffffu;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (k[u] != 0xffffu) {
                const unsigned old = atomicAdd(s_cnt + (k[u] >> 1), 1u << (16 * (k[u] & 1u)));
                s_idx[(old >> (16 * (k[u] & 1u))) & 0xffffu] = (uint16_t)(i0 + u * kScanThreads + t);
            }
    }
    __syncthreads();
    auto end_of = [&](int k) { return (int)s_end[k] + (k >= s_wrap ? 65536 : 0); };
    // 4. means
    float4 *out = a.out + s_base;
    const int sub = lane & 3;
    for (int o0 = w * 8; o0 < (int)total; o0 += kScanThreads / 4) {  // (warp-uniform trip count)
        const int o = o0 + (lane >> 2);
        int f = 0, m = 0;
        if (o < (int)total) {
            const int k = s_list[o];
            f = k > 0 ? end_of(k - 1) : 0;
            m = end_of(k) - f;
            if (m > kGroupLeaf) m = 0;  // a warp's, below
        }
        uint16_t *x = s_idx + f;
        double v[4] = {0, 0, 0, 0};
        Magnitudes g[4];
        for (int i = sub; i < m; i += 16) {  // 4 lanes, 4 points in flight each
            float4 p[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) p[u] = pts[x[min(i + 4 * u, m - 1)]];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (i + 4 * u < m) {
                    v[0] += (double)p[u].x; v[1] += (double)p[u].y; v[2] += (double)p[u].z; v[3] += (double)p[u].w;
                    g[0].take(p[u].x); g[1].take(p[u].y); g[2].take(p[u].z); g[3].take(p[u].w);
                }
        }
        __syncwarp();
        bool exact = true;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
#pragma unroll
            for (int q = 1; q < 4; q <<= 1) {
                v[c] += __shfl_xor_sync(kAll, v[c], q);
                g[c].lo = min(g[c].lo, __shfl_xor_sync(kAll, g[c].lo, q));
                g[c].hi = max(g[c].hi, __shfl_xor_sync(kAll, g[c].hi, q));
            }
            exact = exact && g[c].exact(m);
        }
        if (!__all_sync(kAll, exact || m == 0)) {  // in input order, by the group's first lane
            if (!exact && sub == 0 && m > 0) {
                for (int i = 1; i < m; ++i) {
                    const uint16_t y = x[i];
                    int j = i;
                    for (; j > 0 && x[j - 1] > y; --j) x[j] = x[j - 1];
                    x[j] = y;
                }
                v[0] = v[1] = v[2] = v[3] = 0.0;
                for (int i = 0; i < m; ++i) {
                    const float4 p = pts[x[i]];
                    v[0] += (double)p.x; v[1] += (double)p.y; v[2] += (double)p.z; v[3] += (double)p.w;
                }
            }
            __syncwarp();
#pragma unroll
            for (int c = 0; c < 4; ++c) v[c] = __shfl_sync(kAll, v[c], lane & ~3);
        }
        // (each lane divides one component)
        const double mine = sub == 0 ? v[0] : (sub == 1 ? v[1] : (sub == 2 ? v[2] : v[3]));
        if (m > 0) reinterpret_cast<float *>(out + o)[sub] = (float)(mine / (double)m);
    }
    for (int o0 = w * 32; o0 < (int)total; o0 += kScanThreads) {
        const int ol = o0 + lane;
        const int kl = ol < (int)total ? s_list[ol] : 0;
        const int el = ol < (int)total ? end_of(kl) : 0, fl = ol < (int)total && kl > 0 ? end_of(kl - 1) : 0;
        unsigned big = __ballot_sync(kAll, ol < (int)total && el - fl > kGroupLeaf);
        while (big) {
            const int q = __ffs(big) - 1;
            big &= big - 1u;
            const int k = __shfl_sync(kAll, kl, q), e = __shfl_sync(kAll, el, q), f = __shfl_sync(kAll, fl, q);
            const int m = e - f;
            double s[4] = {0, 0, 0, 0};
            Magnitudes g[4];
            for (int i = f + lane; i < e; i += 32) {
                const float4 p = pts[s_idx[i]];
                s[0] += (double)p.x; s[1] += (double)p.y; s[2] += (double)p.z; s[3] += (double)p.w;
                g[0].take(p.x); g[1].take(p.y); g[2].take(p.z); g[3].take(p.w);
            }
            bool exact = true;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                g[c].lo = __reduce_min_sync(kAll, g[c].lo);
                g[c].hi = __reduce_max_sync(kAll, g[c].hi);
                exact = exact && g[c].exact(m);
#pragma unroll
                for (int x = 16; x > 0; x >>= 1) s[c] += __shfl_xor_sync(kAll, s[c], x);
            }
            if (!exact) {  // in input order
                s[0] = s[1] = s[2] = s[3] = 0.0;
                auto add = [&](float4 p, unsigned in) {  // the points of lanes `in`, in lane order
                    while (in) {
                        const int l = __ffs(in) - 1;
                        in &= in - 1u;
                        s[0] += (double)__shfl_sync(kAll, p.x, l);
                        s[1] += (double)__shfl_sync(kAll, p.y, l);
                        s[2] += (double)__shfl_sync(kAll, p.z, l);
                        s[3] += (double)__shfl_sync(kAll, p.w, l);
                    }
                };
                if (m <= kSortLeaf) {
                    warp_sort(s_idx + f, m);
                    for (int i0 = f; i0 < e; i0 += 32) {
                        const float4 p = pts[s_idx[min(i0 + lane, e - 1)]];
                        add(p, __ballot_sync(kAll, i0 + lane < e));
                    }
                } else {  // most of the scan: its keys in order
                    for (int i0 = 0; i0 < n; i0 += 256) {
                        unsigned x[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u)
                            x[u] = i0 + 32 * u + lane < n ? keys[i0 + 32 * u + lane] : 0xffffu;
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            const unsigned in = __ballot_sync(kAll, x[u] == (unsigned)k);
                            if (in) add(pts[min(i0 + 32 * u + lane, n - 1)], in);
                        }
                    }
                }
            }
            if (lane == 0) out[o0 + q] = mean_of(s[0], s[1], s[2], s[3], m);
        }
    }
}

// key = base[scan] + local leaf key (x fastest); non-finite points get the
// key of the batch's end (sorted last, dropped).
__global__ void key_kernel(const float4 *__restrict__ pts, const int *__restrict__ offsets, int B, float r,
                           const ScanGeom *__restrict__ geom, const int *__restrict__ base, int total_keys, int n,
                           uint32_t *__restrict__ keys) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = pts[i];
    uint32_t k = (uint32_t)total_keys;
    if (finite3(p)) {
        const int b = owner(offsets, B, i);
        const ScanGeom &g = geom[b];
        const long long qx = leaf_of(p.x, r) - g.lo[0], qy = leaf_of(p.y, r) - g.lo[1], qz = leaf_of(p.z, r) - g.lo[2];
        k = (uint32_t)(base[b] + (int)(qx + g.d[0] * (qy + g.d[1] * qz)));
    }
    keys[i] = k;
}

// sorted[j] = pts[order[j]]: the points in key order (one thread per point,
// so the random reads are all in flight at once; writes coalesced).
__global__ void gather_kernel(const float4 *__restrict__ pts, const uint32_t *__restrict__ order, int n,
                              float4 *__restrict__ sorted, const int *__restrict__ sort_err) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < n && !*sort_err) sorted[j] = pts[__ldg(order + j)];
}

// One thread per segment: the FP64 mean of its points in input order (the
// stable sort keeps that order within a segment), written to out[s].
// Segments are in key order (scan, then leaf) and the segment of dropped
// points, if any, is the last, so s is the output index.
__global__ void mean_kernel(const float4 *__restrict__ sorted, const int32_t *__restrict__ seg_start,
                            const uint32_t *__restrict__ seg_key, const int *__restrict__ nseg, int n,
                            uint32_t drop_key, float4 *__restrict__ out) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    const int K = *nseg;
    if (s >= K || seg_key[s] == drop_key) return;
    const int a = seg_start[s], e = s + 1 < K ? seg_start[s + 1] : n;
    double sx = 0, sy = 0, sz = 0, sw = 0;
    for (int j = a; j < e; ++j) {
        const float4 p = sorted[j];
        sx += (double)p.x;
        sy += (double)p.y;
        sz += (double)p.z;
        sw += (double)p.w;
    }
    const double c = (double)(e - a);
    out[s] = make_float4((float)(sx / c), (float)(sy / c), (float)(sz / c), (float)(sw / c));
}

// Output offsets without atomics: scan b's leaves are the segments with keys
// in [base[b], base[b + 1]), so out_off[b] = the number of segments with a
// key below base[b] (a lower bound in the sorted segment keys), b = 0 .. B
// (base[B] = the key total = the dropped points' key).
__global__ void offsets_kernel(const uint32_t *__restrict__ seg_key, const int *__restrict__ nseg,
                               const int *__restrict__ base, int B, int *__restrict__ out_off) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > B) return;
    const uint32_t k = (uint32_t)base[b];
    int lo = 0, hi = *nseg;  // first index in [lo, hi] with seg_key >= k
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (seg_key[mid] < k) lo = mid + 1; else hi = mid;
    }
    out_off[b] = lo;
}

}  // namespace vf

namespace {

struct Buf {
    void *p = nullptr;
    size_t cap = 0;
    cudaError_t ensure(size_t bytes) {
        if (bytes <= cap && p) return cudaSuccess;
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
        cudaError_t e = cudaMalloc(&p, bytes < 256 ? 256 : bytes);
        if (e == cudaSuccess) cap = bytes < 256 ? 256 : bytes;
        return e;
    }
    ~Buf() {
        if (p) cudaFree(p);
    }
};

}  // namespace

struct ndt_filter {
    int device = 0;
    cudaStream_t stream = nullptr;
    Buf geom, base, flags, box, sort_scratch, seg_start, seg_key, sorted, chain, keys;
    int box_cap = 0;
    int *h_flags = nullptr;  // pinned: error flags, key total, largest leaf range and scan; output total, error
    std::string msg;
};

extern "C" {

int ndt_filter_create(int device, ndt_filter **out) {
    if (!out) return NDT_E_ARG;
    *out = nullptr;
    ndt_filter *f = new ndt_filter();
    f->device = device;
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&f->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMallocHost((void **)&f->h_flags, sizeof(int) * 6);
    if (e == cudaSuccess) e = (cudaError_t)ndt::prepare_sort();
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(vf::scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)vf::kScanSmem);
    if (e != cudaSuccess) {
        ndt_filter_destroy(f);
        return NDT_E_CUDA;
    }
    *out = f;
    return NDT_OK;
}

void ndt_filter_destroy(ndt_filter *f) {
    if (!f) return;
    cudaSetDevice(f->device);
    if (f->stream) {
        cudaStreamSynchronize(f->stream);
        cudaStreamDestroy(f->stream);
    }
    if (f->h_flags) cudaFreeHost(f->h_flags);
    delete f;
}

const char *ndt_filter_last_error(const ndt_filter *f) { return f ? f->msg.c_str() : "null filter"; }

void *ndt_filter_stream(ndt_filter *f) { return f ? (void *)f->stream : nullptr; }

#define FCK(call)                                                                  \
    do {                                                                           \
        cudaError_t e_ = (call);                                                   \
        if (e_ != cudaSuccess) {                                                   \
            f->msg = std::string(#call) + ": " + cudaGetErrorString(e_);          \
            return NDT_E_CUDA;                                                     \
        }                                                                          \
    } while (0)

int ndt_voxel_filter_device(ndt_filter *f, int B, const float *d_points, const int *d_offsets, int total_points,
                            float leaf, float *d_out, int *d_out_offsets, int *out_total) {
    ndt::NvtxRange range("voxel filter");
    if (!f || B <= 0 || total_points < 0 || !d_points || !d_offsets || !d_out || !d_out_offsets || !out_total ||
        !(leaf > 0.0f) || !std::isfinite(leaf)) {
        if (f) f->msg = "bad argument";
        return NDT_E_ARG;
    }
    FCK(cudaSetDevice(f->device));
    cudaStream_t st = f->stream;
    const int n = total_points;
    const float r = 1.0f / leaf;
    FCK(f->geom.ensure(sizeof(vf::ScanGeom) * (size_t)B));
    FCK(f->base.ensure(sizeof(int) * (size_t)(B + 1)));
    FCK(f->flags.ensure(sizeof(int) * 4));
    if (f->box_cap < B) {  // the range pass resets the boxes it read; a fresh buffer is set once
        FCK(f->box.ensure(sizeof(long long) * 6 * (size_t)B));
        vf::box_init_kernel<<<(6 * B + 255) / 256, 256, 0, st>>>((long long *)f->box.p, B);
        FCK(cudaGetLastError());
        f->box_cap = B;
    }
    long long *box = (long long *)f->box.p;
    int *base = (int *)f->base.p;
    int *flags = (int *)f->flags.p;
    FCK(cudaMemsetAsync(flags, 0, sizeof(int) * 4, st));
    if (n > 0) {
        const long long warps = ((long long)n + vf::kBoxWarpPoints - 1) / vf::kBoxWarpPoints;
        vf::box_kernel<<<(unsigned)((warps * 32 + vf::kThreads - 1) / vf::kThreads), vf::kThreads, 0, st>>>(
            (const float4 *)d_points, d_offsets, B, n, r, box);
        FCK(cudaGetLastError());
    }
    vf::range_kernel<<<1, vf::kRangeThreads, 0, st>>>(box, B, d_offsets, n, (vf::ScanGeom *)f->geom.p, base, flags);
    FCK(cudaGetLastError());
    FCK(cudaMemcpyAsync(f->h_flags, flags, sizeof(int) * 4, cudaMemcpyDeviceToHost, st));
    FCK(cudaStreamSynchronize(st));
    if (f->h_flags[0]) {
        f->msg = (f->h_flags[0] & 1) ? "a scan spans 2^31 leaves or more" : "the batch spans 2^31 - 1 leaves or more";
        return NDT_E_CAPACITY;
    }
    const int total_keys = f->h_flags[1];  // key total_keys marks the dropped points
    if (n == 0) {
        FCK(cudaMemsetAsync(d_out_offsets, 0, sizeof(int) * (size_t)(B + 1), st));
        FCK(cudaStreamSynchronize(st));
        *out_total = 0;
        return NDT_OK;
    }
    const int leaves = f->h_flags[2] > 0 ? f->h_flags[2] : 1, longest = f->h_flags[3];
    const size_t pts_bytes = sizeof(float4) * (size_t)n, off_bytes = sizeof(int) * (size_t)(B + 1);
    const bool in_place = vf::overlap(d_out, pts_bytes, d_points, pts_bytes) ||
                          vf::overlap(d_out, pts_bytes, d_offsets, off_bytes) ||
                          vf::overlap(d_out_offsets, off_bytes, d_points, pts_bytes) ||
                          vf::overlap(d_out_offsets, off_bytes, d_offsets, off_bytes);
    if (!in_place && vf::scan_fits(leaves, longest) && vf::scan_pays(longest, n)) {
        const size_t head = 256, bytes = head + sizeof(uint64_t) * (size_t)B;
        FCK(f->chain.ensure(bytes));
        FCK(f->keys.ensure(sizeof(uint16_t) * (size_t)n));
        FCK(cudaMemsetAsync(f->chain.p, 0, bytes, st));
        vf::ScanArgs a;
        a.pts = (const float4 *)d_points;
        a.offsets = d_offsets;
        a.geom = (const vf::ScanGeom *)f->geom.p;
        a.r = r;
        a.B = B;
        a.leaves = leaves;
        a.n = longest;
        a.keys = (uint16_t *)f->keys.p;
        a.out = (float4 *)d_out;
        a.out_off = d_out_offsets;
        a.ticket = (int *)f->chain.p;
        a.err = a.ticket + 1;
        a.state = (uint64_t *)((char *)f->chain.p + head);
        vf::scan_kernel<<<B, vf::kScanThreads, vf::scan_smem(leaves, longest), st>>>(a);
        FCK(cudaGetLastError());
        FCK(cudaMemcpyAsync(f->h_flags + 4, d_out_offsets + B, sizeof(int), cudaMemcpyDeviceToHost, st));
        FCK(cudaMemcpyAsync(f->h_flags + 5, a.err, sizeof(int), cudaMemcpyDeviceToHost, st));
        FCK(cudaStreamSynchronize(st));
        if (f->h_flags[5]) {
            f->msg = "a wait between the scans' blocks gave up";
            return NDT_E_CUDA;
        }
        *out_total = f->h_flags[4];
        return NDT_OK;
    }
    int bits = 1;
    while (bits < 32 && (1LL << bits) <= (long long)total_keys) ++bits;
    FCK(f->sort_scratch.ensure(ndt::sort_scratch_bytes(n)));
    FCK(f->seg_start.ensure(sizeof(int32_t) * (size_t)n));
    FCK(f->seg_key.ensure(sizeof(uint32_t) * (size_t)n));
    FCK(f->sorted.ensure(sizeof(float4) * (size_t)n));
    ndt::SortBuffers sb = ndt::sort_buffers(f->sort_scratch.p, n);
    const unsigned pblk = (unsigned)((n + vf::kThreads - 1) / vf::kThreads);
    vf::key_kernel<<<pblk, vf::kThreads, 0, st>>>((const float4 *)d_points, d_offsets, B, r,
                                                  (const vf::ScanGeom *)f->geom.p, base, total_keys, n, sb.k0);
    FCK(cudaGetLastError());
    ndt::sort_segments(sb, n, bits, (int32_t *)f->seg_start.p, (uint32_t *)f->seg_key.p, st, true);
    FCK(cudaGetLastError());
    vf::gather_kernel<<<pblk, vf::kThreads, 0, st>>>((const float4 *)d_points, sb.v0, n, (float4 *)f->sorted.p,
                                                     ndt::sort_error(sb, n));
    vf::mean_kernel<<<pblk, vf::kThreads, 0, st>>>((const float4 *)f->sorted.p, (const int32_t *)f->seg_start.p,
                                                   (const uint32_t *)f->seg_key.p, sb.nseg, n, (uint32_t)total_keys,
                                                   (float4 *)d_out);
    vf::offsets_kernel<<<(B + 1 + vf::kThreads - 1) / vf::kThreads, vf::kThreads, 0, st>>>(
        (const uint32_t *)f->seg_key.p, sb.nseg, base, B, d_out_offsets);
    FCK(cudaGetLastError());
    FCK(cudaMemcpyAsync(f->h_flags + 4, d_out_offsets + B, sizeof(int), cudaMemcpyDeviceToHost, st));
    FCK(cudaMemcpyAsync(f->h_flags + 5, ndt::sort_error(sb, n), sizeof(int), cudaMemcpyDeviceToHost, st));
    FCK(cudaStreamSynchronize(st));
    if (f->h_flags[5]) {
        f->msg = "a wait between the sort's tiles gave up";
        return NDT_E_CUDA;
    }
    *out_total = f->h_flags[4];
    return NDT_OK;
}

}  // extern "C"
