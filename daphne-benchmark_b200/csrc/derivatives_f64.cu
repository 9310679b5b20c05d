// The FP64 derivative pass (precision = 1): every (point, voxel) pair is
// evaluated with the reference's FP64 operations, in its order (updateDerivatives /
// updateHessian, src/CPU/ndt_mapping/kernel.cpp:438-493, 604-649, compat) or the
// Magnusson eq. 6.13 Hessian (corrected), and accumulated in FP64; products with
// structural zeros are left out where the inverse covariance is finite.  The
// neighbour search is the exact one of probe.cuh.  Compiled without
// floating-point contraction, like the reference's x86-64 code.
#include <cuda_runtime.h>
#include <stdint.h>

#include "derivatives.h"
#include "ndt_math.cuh"
#include "probe.cuh"

namespace ndt {

namespace {

constexpr int kSums = 43;  // score, g[6], H[36]

// The pair's contributions to the sums, in the reference's expressions as
// written, or false when it has none.  For voxels whose inverse covariance is
// not finite or beyond 1e30 (kSlotFlag) and points that are not finite (a caller's
// transformed point beside them may be), where a product with a zero of J or h
// can be NaN.
__device__ __noinline__ bool pair_literal(double *out, const double *x, const double *ang, const double *xt,
                                          const double *C, double d1, double d2, bool hess, bool compat) {
    // point derivatives (computePointDerivatives, kernel.cpp:495-560)
    auto dot = [](const double *a, const double *b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; };
    double J[3][6] = {{1, 0, 0, 0, 0, 0}, {0, 1, 0, 0, 0, 0}, {0, 0, 1, 0, 0, 0}};
    J[1][3] = dot(x, ang + 0);
    J[2][3] = dot(x, ang + 3);
    J[0][4] = dot(x, ang + 6);
    J[1][4] = dot(x, ang + 9);
    J[2][4] = dot(x, ang + 12);
    J[0][5] = dot(x, ang + 15);
    J[1][5] = dot(x, ang + 18);
    J[2][5] = dot(x, ang + 21);
    const double *h = ang + 24;
    double blk[6][3];  // a b c d e f
    blk[0][0] = 0; blk[0][1] = dot(x, h + 0); blk[0][2] = dot(x, h + 3);
    blk[1][0] = 0; blk[1][1] = dot(x, h + 6); blk[1][2] = dot(x, h + 9);
    blk[2][0] = 0; blk[2][1] = dot(x, h + 12); blk[2][2] = dot(x, h + 15);
    blk[3][0] = dot(x, h + 18); blk[3][1] = dot(x, h + 21); blk[3][2] = dot(x, h + 24);
    blk[4][0] = dot(x, h + 27); blk[4][1] = dot(x, h + 30); blk[4][2] = dot(x, h + 33);
    blk[5][0] = dot(x, h + 36); blk[5][1] = dot(x, h + 39); blk[5][2] = dot(x, h + 42);
    const int bmap[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
    // updateDerivatives (kernel.cpp:438-493)
    double xCx = C[0] * xt[0] * xt[0] + C[4] * xt[1] * xt[1] + C[8] * xt[2] * xt[2] +
                 (C[1] + C[3]) * xt[0] * xt[1] + (C[2] + C[6]) * xt[0] * xt[2] + (C[5] + C[7]) * xt[1] * xt[2];
    double e = exp(-d2 * (xCx) / 2);
    double score_inc = -d1 * e;
    e = d2 * e;
    if (e > 1 || e < 0 || e != e) return false;
    e *= d1;
    double cov[3];
    for (int i = 0; i < 6; ++i) {
        for (int r = 0; r < 3; ++r) {
            cov[r] = 0;
            for (int c = 0; c < 3; ++c) cov[r] += C[3 * r + c] * J[c][i];
        }
        out[1 + i] = dot(xt, cov) * e;
        if (!hess) continue;
        for (int j = 0; j < 6; ++j) {
            double col[3] = {J[0][j], J[1][j], J[2][j]};
            double hb[3] = {0, 0, 0};
            if (i >= 3 && j >= 3) {
                const double *bb = blk[bmap[i - 3][j - 3]];
                hb[0] = bb[0]; hb[1] = bb[1]; hb[2] = bb[2];
            }
            if (compat) {
                double colh[3] = {col[0] + hb[0], col[1] + hb[1], col[2] + hb[2]};
                double mp[3];
                for (int r = 0; r < 3; ++r) {
                    mp[r] = 0;
                    for (int c = 0; c < 3; ++c) mp[r] += C[3 * r + c] * colh[c];
                }
                out[7 + 6 * i + j] = e * (-d2 * dot(xt, cov) * dot(xt, mp) + dot(col, cov));
            } else {
                double cj[3], ch[3];
                for (int r = 0; r < 3; ++r) {
                    cj[r] = C[3 * r] * col[0] + C[3 * r + 1] * col[1] + C[3 * r + 2] * col[2];
                    ch[r] = C[3 * r] * hb[0] + C[3 * r + 1] * hb[1] + C[3 * r + 2] * hb[2];
                }
                out[7 + 6 * i + j] = e * (-d2 * dot(xt, cov) * dot(xt, cj) + dot(xt, ch) + dot(col, cov));
            }
        }
    }
    out[0] = score_inc;
    return true;
}

// The same for a finite point and inverse covariance, added to A: every sum
// and product that can differ from zero, in the order and with the rounding of
// pair_literal.  Left out are products with the zeros of J and h and the sums
// with them (they change no bit of A: at most the sign of a zero that is added
// to it), and what pair_literal computes for every (i, j) is computed once:
// C J_i (corrected: also C J_j), x' . C J_i and x' . C h_ij.
// About 570 FP64 operations instead of 1800 and no arrays in local memory (the
// loops of pair_literal index them): an evaluation of 33 scans of 1001 to 7001
// points takes 29 us instead of 70 (32 with a full butterfly for each sum at the
// end, see warp_sums).  Bound by latency: the sums and one pair's terms fill the
// registers of 8 warps an SM (two blocks of 128 registers a thread, which spill
// 1 KB: 22% slower).
template <bool COMPAT>
__device__ __forceinline__ void add_pair_fp64(double (&A)[kSums], double x0, double x1, double x2, const double *ang,
                                              double p0, double p1, double p2, const double (&C)[9], double d1,
                                              double d2, bool hess) {
    const double xCx = C[0] * p0 * p0 + C[4] * p1 * p1 + C[8] * p2 * p2 + (C[1] + C[3]) * p0 * p1 +
                       (C[2] + C[6]) * p0 * p2 + (C[5] + C[7]) * p1 * p2;
    double e = exp(-d2 * (xCx) / 2);
    const double score_inc = -d1 * e;
    e = d2 * e;
    if (e > 1 || e < 0 || e != e) return;
    e *= d1;
    auto dot = [&](const double *b) { return x0 * b[0] + x1 * b[1] + x2 * b[2]; };
    // column j >= 3 of J: (j0, j1, j2)[j - 3], its first entry 0 for j = 3
    const double j0[3] = {0, dot(ang + 6), dot(ang + 15)};
    const double j1[3] = {dot(ang + 0), dot(ang + 9), dot(ang + 18)};
    const double j2[3] = {dot(ang + 3), dot(ang + 12), dot(ang + 21)};
    // C J_i, its row r at [r]; x' . C J_i
    auto row = [&](int r, bool first, double v0, double v1, double v2) {
        return first ? C[3 * r] * v0 + C[3 * r + 1] * v1 + C[3 * r + 2] * v2 : C[3 * r + 1] * v1 + C[3 * r + 2] * v2;
    };
    double cov[6][3], a[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
#pragma unroll
        for (int r = 0; r < 3; ++r)
            cov[i][r] = i < 3 ? C[3 * r + i] : row(r, i > 3, j0[i < 3 ? 0 : i - 3], j1[i < 3 ? 0 : i - 3], j2[i < 3 ? 0 : i - 3]);
        a[i] = p0 * cov[i][0] + p1 * cov[i][1] + p2 * cov[i][2];
        A[1 + i] += a[i] * e;
    }
    A[0] += score_inc;
    if (!hess) return;
    const double *h = ang + 24;
    // point-Hessian vectors a b c (first entry 0), d e f
    double b[6];           // corrected: x' . C h
    double hv[6][3];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        hv[k][0] = k < 3 ? 0.0 : dot(h + 18 + 9 * (k < 3 ? 0 : k - 3));
        hv[k][1] = k < 3 ? dot(h + 6 * k) : dot(h + 21 + 9 * (k < 3 ? 0 : k - 3));
        hv[k][2] = k < 3 ? dot(h + 6 * k + 3) : dot(h + 24 + 9 * (k < 3 ? 0 : k - 3));
        if (!COMPAT)
            b[k] = p0 * row(0, k >= 3, hv[k][0], hv[k][1], hv[k][2]) + p1 * row(1, k >= 3, hv[k][0], hv[k][1], hv[k][2]) +
                   p2 * row(2, k >= 3, hv[k][0], hv[k][1], hv[k][2]);
    }
    constexpr int bmap[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const double da = -d2 * a[i];
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            const int jj = j < 3 ? 0 : j - 3, ii = i < 3 ? 0 : i - 3;
            // J_j . C J_i
            const double jc = j < 3 ? cov[i][j < 3 ? j : 0]
                                    : (j == 3 ? j1[jj] * cov[i][1] + j2[jj] * cov[i][2]
                                              : j0[jj] * cov[i][0] + j1[jj] * cov[i][1] + j2[jj] * cov[i][2]);
            const bool both = i >= 3 && j >= 3;
            const int k = bmap[ii][jj];
            double v;
            if (COMPAT) {  // x' . C (J_j + h_ij)
                double am = a[j];
                if (both) {
                    const bool first = j > 3 || k >= 3;
                    const double c0 = j > 3 ? (k >= 3 ? j0[jj] + hv[k][0] : j0[jj]) : hv[k][0];
                    const double c1 = j1[jj] + hv[k][1], c2 = j2[jj] + hv[k][2];
                    am = p0 * row(0, first, c0, c1, c2) + p1 * row(1, first, c0, c1, c2) +
                         p2 * row(2, first, c0, c1, c2);
                }
                v = da * am + jc;
            } else {
                v = both ? da * a[j] + b[k] + jc : da * a[j] + jc;
            }
            A[7 + 6 * i + j] += e * v;
        }
    }
}

// The warp's sums of A[k] over its lanes, to out[k]: the butterfly over lane
// distances 16, 8, 4, 2, 1 (both sides of an exchange add the same two numbers,
// so every lane of a full butterfly holds the same bits), with each exchange
// halving the values that a lane still carries: 44 double exchanges, not 215.
__device__ __forceinline__ void warp_sums(double (&A)[kSums], int lane, double *out) {
    int n = kSums, base = 0, end = kSums;  // this lane carries values base .. min(base + n, end) - 1
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const int h = (n + 1) / 2;  // the lane without the bit keeps the first h
        const bool upper = lane & o;
#pragma unroll
        for (int k = 0; k < kSums; ++k) {
            if (k < h) {
                const double lo = A[k], hi = k + h < n ? A[k + h] : 0.0;
                A[k] = (upper ? hi : lo) + __shfl_xor_sync(kFull, upper ? lo : hi, o);
            }
        }
        if (upper) base += h;
        else end = min(end, base + h);
        n = h;
    }
#pragma unroll
    for (int k = 0; k < 2; ++k)
        if (base + k < end) out[base + k] = A[k];
}

constexpr int kTile64 = 256;

template <bool COMPAT>
__global__ void __launch_bounds__(kTile64, 1) derivative_f64_kernel(const __grid_constant__ EvalArgs args) {
    constexpr int kW = kTile64 / 32;
    __shared__ float s_T[12];
    __shared__ double s_ang[kAngle];
    __shared__ int s_mode;
    __shared__ float s_pts[kW][6][32];  // original xyz, transformed xyz
    __shared__ unsigned s_list[kW][kList];
    __shared__ double s_red[kW][kSums];
    __shared__ unsigned s_cnt[kW][3];

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const GridDev &grid = args.grid;
    unsigned *list = s_list[warp];
    float (*pts)[32] = s_pts[warp];

    for (int ti = blockIdx.x, nt = *args.num_tiles; ti < nt; ti += gridDim.x) {
        const Tile tile = args.tiles[ti];
        const AlignState *st = args.states + tile.align;
        __syncthreads();
        if (threadIdx.x == 0) s_mode = st->eval_mode;
        if (threadIdx.x < 12) s_T[threadIdx.x] = st->T[threadIdx.x];
        if (threadIdx.x < kAngle) s_ang[threadIdx.x] = st->angd[threadIdx.x];
        __syncthreads();
        const int mode = s_mode;
        if (mode == kEvalNone) continue;
        const bool hess = eval_level(mode) == kLevelHessian;
        const int i = tile.start + threadIdx.x;
        const bool valid = i < tile.end;
        const float4 x = valid ? args.points[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        float px, py, pz;
        if (args.trans) {
            const float4 y = valid ? args.trans[i] : make_float4(0.f, 0.f, 0.f, 0.f);
            px = y.x; py = y.y; pz = y.z;
        } else {
            px = transform_row(s_T, x.x, x.y, x.z);
            py = transform_row(s_T + 4, x.x, x.y, x.z);
            pz = transform_row(s_T + 8, x.x, x.y, x.z);
        }
        __syncwarp();
        pts[0][lane] = x.x; pts[1][lane] = x.y; pts[2][lane] = x.z;
        pts[3][lane] = px; pts[4][lane] = py; pts[5][lane] = pz;
        const unsigned literal = __ballot_sync(kFull, !(isfinite(x.x) && isfinite(x.y) && isfinite(x.z)));
        double A[kSums];
#pragma unroll
        for (int k = 0; k < kSums; ++k) A[k] = 0.0;
        unsigned n_probe = 0, n_occ = 0, n_pair = 0;
        auto consume = [&](int n) {
            for (int base = 0; base < n; base += 32) {
                const int kk = base + lane;
                if (kk >= n) break;
                const unsigned code = list[kk];
                const int owner = code & 31;
                const int slot = (int)(code >> 6);
                const double4 m = ldg_d4(grid.mean + slot);
                const double x0 = pts[0][owner], x1 = pts[1][owner], x2 = pts[2][owner];
                const double p0 = (double)pts[3][owner] - m.x, p1 = (double)pts[4][owner] - m.y,
                             p2 = (double)pts[5][owner] - m.z;
                const double *icov = grid.icov64 + 9 * (size_t)slot;
                if ((code & 32u) || ((literal >> owner) & 1u)) {
                    const double xo[3] = {x0, x1, x2}, xt[3] = {p0, p1, p2};
                    double c[kSums];
                    if (pair_literal(c, xo, s_ang, xt, icov, args.d1, args.d2, hess, COMPAT)) {
#pragma unroll
                        for (int k = 0; k < kSums; ++k)
                            if (k < 7 || hess) A[k] += c[k];
                    }
                } else {
                    double C[9];
#pragma unroll
                    for (int k = 0; k < 9; ++k) C[k] = __ldg(icov + k);
                    add_pair_fp64<COMPAT>(A, x0, x1, x2, s_ang, p0, p1, p2, C, args.d1, args.d2, hess);
                }
                ++n_pair;
            }
        };
        int resume = 0;
        do {
            __syncwarp();
            ListSink sink{list, 0};
            collect_pairs(grid, px, py, pz, valid, sink, n_probe, n_occ, resume);
            __syncwarp();
            consume(sink.n);
        } while (resume >= 0);
        warp_sums(A, lane, s_red[warp]);
        for (int o = 16; o > 0; o >>= 1) {
            n_probe += __shfl_xor_sync(kFull, n_probe, o);
            n_occ += __shfl_xor_sync(kFull, n_occ, o);
            n_pair += __shfl_xor_sync(kFull, n_pair, o);
        }
        if (lane == 0) {
            s_cnt[warp][0] = n_probe;
            s_cnt[warp][1] = n_occ;
            s_cnt[warp][2] = n_pair;
        }
        __syncthreads();
        double *out = args.partials + (size_t)tile.slot * kPartial;
        if (threadIdx.x < kPartial) {
            const int k = threadIdx.x;
            double v = 0.0;
            if (k < kSums) {
                for (int w = 0; w < kW; ++w) v += s_red[w][k];
            } else {
                unsigned np = 0;
                for (int w = 0; w < kW; ++w) np += s_cnt[w][2];
                v = (double)np;
            }
            out[k] = v;
        }
        if (threadIdx.x == 0 && args.counters) {
            unsigned long long a0 = 0, a1 = 0, a2 = 0;
            for (int w = 0; w < kW; ++w) {
                a0 += s_cnt[w][0];
                a1 += s_cnt[w][1];
                a2 += s_cnt[w][2];
            }
            atomicAdd(&args.counters->probes, a0);
            atomicAdd(&args.counters->occupied_probes, a1);
            atomicAdd(&args.counters->pairs, a2);
            atomicAdd(&args.counters->points, (unsigned long long)(tile.end - tile.start));
            atomicAdd(&args.counters->tiles, 1ull);
        }
    }
}

}  // namespace

int launch_derivatives_f64(const EvalArgs &args, int sms, cudaStream_t st) {
    if (args.tile_size != kTile64) return (int)cudaErrorInvalidValue;
    int blocks = sms < args.max_tiles ? sms : args.max_tiles;
    if (args.compat)
        derivative_f64_kernel<true><<<blocks, kTile64, 0, st>>>(args);
    else
        derivative_f64_kernel<false><<<blocks, kTile64, 0, st>>>(args);
    return (int)cudaGetLastError();
}

}  // namespace ndt
