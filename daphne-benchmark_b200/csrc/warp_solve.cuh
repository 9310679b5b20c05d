// The 6x6 solve of a Newton step by one warp.
#pragma once
#include <cuda_runtime.h>

namespace ndt {

// solve6 (ndt_math.cuh) of H x = -g with row r of the system in lane r < 6:
// the same pivots and the same operations on the entries that are read again,
// the rows of a column in parallel; x in every lane.
__device__ __forceinline__ void warp_solve6(const double *H, const double *g, double *x) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int r = lane < 6 ? lane : 5;
    double a[6], b = -g[r];
#pragma unroll
    for (int k = 0; k < 6; ++k) a[k] = H[6 * r + k];
    int at[6] = {0, 1, 2, 3, 4, 5};  // the lane whose row is at each position
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        const double m = fabs(a[j]);
        double mx = __shfl_sync(kAll, m, at[j]);
        int mi = j;
#pragma unroll
        for (int i = j + 1; i < 6; ++i) {
            const double v = __shfl_sync(kAll, m, at[i]);
            if (v > mx) {
                mi = i;
                mx = v;
            }
        }
#pragma unroll
        for (int i = j + 1; i < 6; ++i)
            if (mi == i) {
                const int t = at[i];
                at[i] = at[j];
                at[j] = t;
                // (the reference swaps the rows of A only: b stays at its position)
                b = __shfl_sync(kAll, b, lane == at[i] ? at[j] : (lane == at[j] ? at[i] : lane));
            }
        if (mx == 0.0 && lane == at[j]) a[j] = 0.001;
        bool below = false;
#pragma unroll
        for (int i = j + 1; i < 6; ++i) below |= lane == at[i];
        if (j == 5) break;
        const double pj = __shfl_sync(kAll, a[j], at[j]);
        const double piv = a[j] / pj;
#pragma unroll
        for (int k = j + 1; k < 6; ++k) {
            const double t = a[k] - piv * __shfl_sync(kAll, a[k], at[j]);
            if (below) a[k] = t;
        }
        const double t = b - piv * __shfl_sync(kAll, b, at[j]);
        if (below) b = t;
    }
#pragma unroll
    for (int i = 5; i >= 0; --i) {
        double sum = 0.0;
#pragma unroll
        for (int j = i + 1; j < 6; ++j) sum = sum + a[j] * x[j];
        const double xi = i == 5 ? b / a[5] : (b - sum) / a[i];
        x[i] = __shfl_sync(kAll, xi, at[i]);
    }
}

}  // namespace ndt
