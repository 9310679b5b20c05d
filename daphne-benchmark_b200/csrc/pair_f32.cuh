// FP32 pair evaluation of the derivative pass, shared by its two kernels
// (derivatives_f32.cu, derivatives_wide.cu), which are compiled with
// floating-point contraction.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "derivatives.h"
#include "probe.cuh"

namespace ndt {

// ---------------------------------------------------------------------------
// FP32 pair evaluation, factored through the point.
//
// For a point x with Jacobian J (3 x 6; columns e0, e1, e2, J_3, J_4, J_5) and
// point-Hessian vectors h_ij (i, j >= 3), the pairs (x, voxel v) contribute,
// with x' = x_trans - mean_v, C = C_v, q = C x', e = exp(-d2 x'^T q / 2),
// w = d1 d2 e (kept when 0 <= d2 e <= 1, kernel.cpp:456) and a_i = q . J_i:
//   score   sum -d1 e
//   g_i     sum w a_i                              = J_i . U
//   S_ij    sum w (-d2 a_i a_j + J_j^T C J_i)      = J_i^T (W - d2 Q) J_j
//   R_ij    compat:    sum w a_i (q . h_ij)        = J_i^T Q h_ij
//           corrected: sum w (q . h_ij)            = U . h_ij
// with the point's sums U = sum w q, Q = sum w q q^T, W = sum w C.  A pair
// therefore costs 16 FMA-type sums (PairSums) and a point one contraction
// with its J and h (contract_add), however many pairs it has.  H = S + k R,
// k = -d2 (compat, the reference's :486-488 form) or 1 (corrected, Magnusson
// eq. 6.13), is assembled from the block totals.
struct PairSums {
    float s, u0, u1, u2;
    float q00, q01, q02, q11, q12, q22;
    float w00, w01, w02, w11, w12, w22;
};

__device__ __forceinline__ void zero(PairSums &F) {
    F.s = F.u0 = F.u1 = F.u2 = 0.0f;
    F.q00 = F.q01 = F.q02 = F.q11 = F.q12 = F.q22 = 0.0f;
    F.w00 = F.w01 = F.w02 = F.w11 = F.w12 = F.w22 = 0.0f;
}

__device__ __forceinline__ void pair_sums(PairSums &F, float p0, float p1, float p2, float c00, float c01, float c02,
                                          float c11, float c12, float c22, float d1, float d2, int level) {
    const float q0 = fmaf(c00, p0, fmaf(c01, p1, c02 * p2));
    const float q1 = fmaf(c01, p0, fmaf(c11, p1, c12 * p2));
    const float q2 = fmaf(c02, p0, fmaf(c12, p1, c22 * p2));
    const float xCx = fmaf(p0, q0, fmaf(p1, q1, p2 * q2));
    const float e = expf(-d2 * xCx * 0.5f);
    const float e2 = d2 * e;
    if (!(e2 <= 1.0f && e2 >= 0.0f)) return;  // kernel.cpp:456 (also rejects NaN)
    F.s = fmaf(-d1, e, F.s);
    if (level == kLevelScore) return;
    const float w = d1 * e2;
    // every multiply-add is written as fmaf or as separately rounded
    // operations, so the FP32 results do not depend on the compiler's
    // contraction choices (which can change with the surrounding code)
    const float wq0 = __fmul_rn(w, q0), wq1 = __fmul_rn(w, q1), wq2 = __fmul_rn(w, q2);
    F.u0 = fmaf(w, q0, F.u0);
    F.u1 = fmaf(w, q1, F.u1);
    F.u2 = fmaf(w, q2, F.u2);
    if (level != kLevelHessian) return;
    F.q00 = fmaf(wq0, q0, F.q00);
    F.q01 = fmaf(wq0, q1, F.q01);
    F.q02 = fmaf(wq0, q2, F.q02);
    F.q11 = fmaf(wq1, q1, F.q11);
    F.q12 = fmaf(wq1, q2, F.q12);
    F.q22 = fmaf(wq2, q2, F.q22);
    F.w00 = fmaf(w, c00, F.w00);
    F.w01 = fmaf(w, c01, F.w01);
    F.w02 = fmaf(w, c02, F.w02);
    F.w11 = fmaf(w, c11, F.w11);
    F.w12 = fmaf(w, c12, F.w12);
    F.w22 = fmaf(w, c22, F.w22);
}

// Symmetric 3 x 3 (m00 m01 m02 m11 m12 m22) times v.
__device__ __forceinline__ void sym_mul(float m00, float m01, float m02, float m11, float m12, float m22, float v0,
                                        float v1, float v2, float &r0, float &r1, float &r2) {
    r0 = fmaf(m00, v0, fmaf(m01, v1, m02 * v2));
    r1 = fmaf(m01, v0, fmaf(m11, v1, m12 * v2));
    r2 = fmaf(m02, v0, fmaf(m12, v1, m22 * v2));
}

// A point's contribution (its PairSums F contracted with its J and h), added
// to (ADD) or stored in the lane's acc[k * stride]: [0] score, [1..6] g,
// [7..27] S (upper triangle), [28..36] R (compat: 3 x 3; corrected: the upper
// triangle only).
// ang = the alignment's FP32 angle terms (j_ang a..h, h_ang a2..f3, 3 each).
template <bool ADD>
__device__ __forceinline__ void contract(const PairSums &F, float x0, float x1, float x2, const float *ang,
                                         float *acc, int stride, float d2, int level, bool compat) {
    auto put = [](float *p, float v) { *p = ADD ? *p + v : v; };
    put(acc, F.s);
    if (level == kLevelScore) return;
    // J_3 = (0, J13, J23), J_4 = (J04, J14, J24), J_5 = (J05, J15, J25)
    // (computePointDerivatives, kernel.cpp:512-521)
    const float J13 = dot3f(x0, x1, x2, ang + 0), J23 = dot3f(x0, x1, x2, ang + 3);
    const float J04 = dot3f(x0, x1, x2, ang + 6), J14 = dot3f(x0, x1, x2, ang + 9);
    const float J24 = dot3f(x0, x1, x2, ang + 12), J05 = dot3f(x0, x1, x2, ang + 15);
    const float J15 = dot3f(x0, x1, x2, ang + 18), J25 = dot3f(x0, x1, x2, ang + 21);
    put(acc + 1 * stride, F.u0);
    put(acc + 2 * stride, F.u1);
    put(acc + 3 * stride, F.u2);
    put(acc + 4 * stride, fmaf(J13, F.u1, J23 * F.u2));
    put(acc + 5 * stride, fmaf(J04, F.u0, fmaf(J14, F.u1, J24 * F.u2)));
    put(acc + 6 * stride, fmaf(J05, F.u0, fmaf(J15, F.u1, J25 * F.u2)));
    if (level != kLevelHessian) return;
    // P = W - d2 Q
    const float nd2 = -d2;
    const float P00 = fmaf(nd2, F.q00, F.w00), P01 = fmaf(nd2, F.q01, F.w01), P02 = fmaf(nd2, F.q02, F.w02);
    const float P11 = fmaf(nd2, F.q11, F.w11), P12 = fmaf(nd2, F.q12, F.w12), P22 = fmaf(nd2, F.q22, F.w22);
    float a0, a1, a2, b0, b1, b2, c0, c1, c2;  // P J_3, P J_4, P J_5
    sym_mul(P00, P01, P02, P11, P12, P22, 0.0f, J13, J23, a0, a1, a2);
    sym_mul(P00, P01, P02, P11, P12, P22, J04, J14, J24, b0, b1, b2);
    sym_mul(P00, P01, P02, P11, P12, P22, J05, J15, J25, c0, c1, c2);
    float *S = acc + 7 * stride;  // sidx order: (0,0..5), (1,1..5), (2,2..5), (3,3..5), (4,4..5), (5,5)
    put(S + 0 * stride, P00);
    put(S + 1 * stride, P01);
    put(S + 2 * stride, P02);
    put(S + 3 * stride, a0);
    put(S + 4 * stride, b0);
    put(S + 5 * stride, c0);
    put(S + 6 * stride, P11);
    put(S + 7 * stride, P12);
    put(S + 8 * stride, a1);
    put(S + 9 * stride, b1);
    put(S + 10 * stride, c1);
    put(S + 11 * stride, P22);
    put(S + 12 * stride, a2);
    put(S + 13 * stride, b2);
    put(S + 14 * stride, c2);
    put(S + 15 * stride, fmaf(J13, a1, J23 * a2));
    put(S + 16 * stride, fmaf(J13, b1, J23 * b2));
    put(S + 17 * stride, fmaf(J13, c1, J23 * c2));
    put(S + 18 * stride, fmaf(J04, b0, fmaf(J14, b1, J24 * b2)));
    put(S + 19 * stride, fmaf(J04, c0, fmaf(J14, c1, J24 * c2)));
    put(S + 20 * stride, fmaf(J05, c0, fmaf(J15, c1, J25 * c2)));
    // point-Hessian vectors (computePointDerivatives, kernel.cpp:523-558):
    // h33 = (0, a2, a3), h34 = (0, b2, b3), h35 = (0, c2, c3), h44 = d,
    // h45 = e, h55 = f
    const float *h = ang + 24;
    const float h33y = dot3f(x0, x1, x2, h + 0), h33z = dot3f(x0, x1, x2, h + 3);
    const float h34y = dot3f(x0, x1, x2, h + 6), h34z = dot3f(x0, x1, x2, h + 9);
    const float h35y = dot3f(x0, x1, x2, h + 12), h35z = dot3f(x0, x1, x2, h + 15);
    const float h44x = dot3f(x0, x1, x2, h + 18), h44y = dot3f(x0, x1, x2, h + 21), h44z = dot3f(x0, x1, x2, h + 24);
    const float h45x = dot3f(x0, x1, x2, h + 27), h45y = dot3f(x0, x1, x2, h + 30), h45z = dot3f(x0, x1, x2, h + 33);
    const float h55x = dot3f(x0, x1, x2, h + 36), h55y = dot3f(x0, x1, x2, h + 39), h55z = dot3f(x0, x1, x2, h + 42);
    float *R = acc + 28 * stride;
    if (compat) {
        // R[a][b] = J_{3+a} . (Q h_{3+a,3+b})
        float t0, t1, t2;
        sym_mul(F.q00, F.q01, F.q02, F.q11, F.q12, F.q22, 0.0f, h33y, h33z, t0, t1, t2);
        put(R, fmaf(J13, t1, J23 * t2));
        sym_mul(F.q00, F.q01, F.q02, F.q11, F.q12, F.q22, 0.0f, h34y, h34z, t0, t1, t2);
        put(R + 1 * stride, fmaf(J13, t1, J23 * t2));
        put(R + 3 * stride, fmaf(J04, t0, fmaf(J14, t1, J24 * t2)));
        sym_mul(F.q00, F.q01, F.q02, F.q11, F.q12, F.q22, 0.0f, h35y, h35z, t0, t1, t2);
        put(R + 2 * stride, fmaf(J13, t1, J23 * t2));
        put(R + 6 * stride, fmaf(J05, t0, fmaf(J15, t1, J25 * t2)));
        sym_mul(F.q00, F.q01, F.q02, F.q11, F.q12, F.q22, h44x, h44y, h44z, t0, t1, t2);
        put(R + 4 * stride, fmaf(J04, t0, fmaf(J14, t1, J24 * t2)));
        sym_mul(F.q00, F.q01, F.q02, F.q11, F.q12, F.q22, h45x, h45y, h45z, t0, t1, t2);
        put(R + 5 * stride, fmaf(J04, t0, fmaf(J14, t1, J24 * t2)));
        put(R + 7 * stride, fmaf(J05, t0, fmaf(J15, t1, J25 * t2)));
        sym_mul(F.q00, F.q01, F.q02, F.q11, F.q12, F.q22, h55x, h55y, h55z, t0, t1, t2);
        put(R + 8 * stride, fmaf(J05, t0, fmaf(J15, t1, J25 * t2)));
    } else {
        // R[a][b] = U . h_{3+a,3+b}, a <= b
        put(R, fmaf(F.u1, h33y, F.u2 * h33z));
        put(R + 1 * stride, fmaf(F.u1, h34y, F.u2 * h34z));
        put(R + 2 * stride, fmaf(F.u1, h35y, F.u2 * h35z));
        put(R + 4 * stride, fmaf(F.u0, h44x, fmaf(F.u1, h44y, F.u2 * h44z)));
        put(R + 5 * stride, fmaf(F.u0, h45x, fmaf(F.u1, h45y, F.u2 * h45z)));
        put(R + 8 * stride, fmaf(F.u0, h55x, fmaf(F.u1, h55y, F.u2 * h55z)));
    }
}

__device__ __forceinline__ int level_values(int level) {
    return level == kLevelScore ? 1 : (level == kLevelGradient ? 7 : kAcc);
}

// Chunks of this pass, and the k-th of them: of the active list (large chunks
// from its front, small ones from its back, so that the small ones come last),
// or of all chunks.
__device__ __forceinline__ int pass_chunks(const EvalArgs &args) {
    return args.active_chunks ? args.num_active[0] + args.num_active[1] : *args.num_chunks;
}
__device__ __forceinline__ int active_chunk(const EvalArgs &args, int k) {
    if (!args.active_chunks) return k;
    const int nb = args.num_active[0];
    return args.active_chunks[k < nb ? k : args.active_capacity - 1 - (k - nb)];
}

// Queues a pair with a flagged voxel for flagged_kernel (FP64).
__device__ __forceinline__ void queue_flagged(const EvalArgs &args, int align, int point, int slot) {
    const unsigned q = atomicAdd(args.flag_n, 1u);
    if (q < args.flag_cap) args.flag_q[q] = make_int4(align, point, slot, 0);
}

// x' = x_trans - mean (kernel.cpp:692-694) from the (hi, lo) float split of
// the FP64 mean, and the pair's sums.
__device__ __forceinline__ void add_pair(const GridDev &g, PairSums &F, int slot, float px, float py, float pz, float d1,
                                         float d2, int level) {
    const float4 *r = g.vox32 + 3 * slot;  // one 48-byte record
    const float4 hi = __ldg(r), lo = __ldg(r + 1), cc = __ldg(r + 2);
    const float p0 = __fsub_rn(__fsub_rn(px, hi.x), lo.x);
    const float p1 = __fsub_rn(__fsub_rn(py, hi.y), lo.y);
    const float p2 = __fsub_rn(__fsub_rn(pz, hi.z), lo.z);
    pair_sums(F, p0, p1, p2, hi.w, lo.w, cc.x, cc.y, cc.z, cc.w, d1, d2, level);
}

}  // namespace ndt
