// Per-alignment control on the device: set-up from the guess, the Newton /
// More-Thuente state machine between derivative passes, and the result write.
//
// The reference runs, per alignment (computeTransformation,
// src/CPU/ndt_mapping/kernel.cpp:1175-1272, computeStepLengthMT :1015-1144):
//   eval(guess) ; repeat { solve ; step length (1 + <= 10 line-search evals +
//   optional Hessian pass) ; pose update ; convergence test }.
// Here every alignment of a batch is a small state machine in AlignState; a
// round is one derivative pass over all tiles of the alignments that asked for
// an evaluation, then one step_kernel call in which each such alignment
// consumes its result and advances until it needs the next evaluation (or is
// done).  All control arithmetic is FP64 with the reference's operation order.
#include <cuda_runtime.h>
#include <stdint.h>

#include "align.h"
#include "ndt_math.cuh"
#include "warp_solve.cuh"

namespace ndt {

namespace {

constexpr double kMu = 1.e-4;     // sufficient decrease (kernel.cpp:1042)
constexpr double kNu = 0.9;       // curvature condition (kernel.cpp:1044)
constexpr int kMaxStepIterations = 10;  // kernel.cpp:1039

// What one warp needs to step an alignment: the state's copy in shared memory
// and the cosines and sines of its angles (3) and half angles (3).
struct StepSmem {
    AlignState st;
    double c[6], s[6];
    double v[kPartial];  // the evaluation's sums
};

__device__ __forceinline__ int bcast0(int v) { return __shfl_sync(0xffffffffu, v, 0); }

// The cosines and sines of pose p's angles, one angle per lane (the whole
// warp calls this and the three functions below).
__device__ __forceinline__ void warp_trig(StepSmem &m, const double *p) {
    const int lane = threadIdx.x & 31;
    if (lane < 6) {
        const double a = p[3 + lane % 3];
        const double x = lane < 3 ? a : half_angle(a);
        m.c[lane] = cos(x);
        m.s[lane] = sin(x);
    }
    __syncwarp();
}

// The angle terms of pose p, after warp_trig.
__device__ __forceinline__ void warp_angles(StepSmem &m, const double *p, bool compat) {
    const int lane = threadIdx.x & 31;
    if (lane == 0) angle_terms(p, m.c, m.s, m.st.angd, compat);
    __syncwarp();
    for (int k = lane; k < kAngle; k += 32) m.st.angf[k] = (float)m.st.angd[k];
}

// The transform and the angle terms of the trial pose.
__device__ __forceinline__ void warp_set_pose(StepSmem &m, const StepParams &P) {
    warp_trig(m, m.st.x_t);
    if ((threadIdx.x & 31) == 1) {  // (beside the angle terms, which lane 0 writes)
        if (P.compat)
            build_tm_compat(m.st.T, m.c + 3, m.s + 3);
        else
            build_tm_corrected(m.st.T, m.st.x_t, m.c, m.s);
    }
    warp_angles(m, m.st.x_t, P.compat != 0);
    __syncwarp();
}

__device__ __forceinline__ double dot6(const double *a, const double *b) {
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2] + a[3] * b[3] + a[4] * b[4] + a[5] * b[5];
}

// Request an evaluation, unless the watchdog budget is spent.
__device__ bool request(AlignState &s, const StepParams &P, int mode, int phase) {
    if (s.evals >= P.watchdog_evals) {
        s.status = NDT_ST_WATCHDOG_DEV;
        s.converged = 0;
        s.phase = kPhaseDone;
        s.eval_mode = kEvalNone;
        return false;
    }
    s.eval_mode = mode;
    s.phase = phase;
    return true;
}

// What lane 0 leaves the warp to do next.
enum StepAct : int {
    kActNone = 0,    // nothing: an evaluation is requested or the alignment is done
    kActPose = 1,    // set the trial pose, then request evaluation `mode` in `phase`
    kActNewton = 2,  // start a Newton iteration
    kActEnd = 3,     // the step ended without an evaluation: newton_end
};

// Start of a Newton iteration from its step dp (kernel.cpp:1214-1245) and of
// the step-length search up to its first evaluation (:1019-1066).
__device__ int newton_start(AlignState &s, const StepParams &P, const double *dp) {
    double norm = sqrt(dp[0] * dp[0] + dp[1] * dp[1] + dp[2] * dp[2] + dp[3] * dp[3] + dp[4] * dp[4] + dp[5] * dp[5]);
    if (P.compat) norm = 1;  // kernel.cpp:1231
    if (norm == 0 || norm != norm) {
        s.converged = norm == norm;
        s.phase = kPhaseDone;
        s.eval_mode = kEvalNone;
        return kActNone;
    }
    for (int i = 0; i < 6; ++i) s.dir[i] = dp[i] / norm;
    // computeStepLengthMT(p, dir, step_init = norm, step_max, step_min)
    s.phi_0 = -s.score;
    s.d_phi_0 = -(dot6(s.g, s.dir));
    if (s.d_phi_0 >= 0) {
        if (s.d_phi_0 == 0) {
            s.a_t = 0;  // not a descent direction: step 0, no evaluation
            return kActEnd;
        }
        s.d_phi_0 *= -1;
        for (int i = 0; i < 6; ++i) s.dir[i] *= -1;
    }
    s.step_iterations = 0;
    s.a_l = 0;
    s.a_u = 0;
    s.f_l = psi_mt(s.a_l, s.phi_0, s.phi_0, s.d_phi_0, kMu);
    s.g_l = dpsi_mt(s.d_phi_0, s.d_phi_0, kMu);
    s.f_u = psi_mt(s.a_u, s.phi_0, s.phi_0, s.d_phi_0, kMu);
    s.g_u = dpsi_mt(s.d_phi_0, s.d_phi_0, kMu);
    // the reference tests "> 0" (kernel.cpp:1053), which skips the search
    // whenever step_max > step_min; the corrected NDT tests "< 0"
    s.interval_converged = P.compat ? (s.step_max - s.step_min) > 0 : (s.step_max - s.step_min) < 0;
    s.open_interval = 1;
    double a_t = norm;
    a_t = std_min(a_t, s.step_max);
    a_t = std_max(a_t, s.step_min);
    s.a_t = a_t;
    for (int i = 0; i < 6; ++i) s.x_t[i] = s.p[i] + s.dir[i] * a_t;
    return kActPose;
}

// Pose update and convergence test after a step (kernel.cpp:1246-1266).
// Returns true when the alignment is done.
__device__ bool newton_end(AlignState &s, const StepParams &P) {
    double dp[6];
    for (int i = 0; i < 6; ++i) dp[i] = s.dir[i] * s.a_t;
    for (int i = 0; i < 6; ++i) s.p[i] = s.p[i] + dp[i];
    if (s.nr_iterations > P.max_iterations || (s.nr_iterations && (fabs(s.a_t) < P.eps))) s.converged = 1;
    s.nr_iterations++;
    if (s.converged) {
        s.phase = kPhaseDone;
        s.eval_mode = kEvalNone;
        return true;
    }
    return false;
}

// Loop test of the line search (kernel.cpp:1076) and its next trial point
// (:1078-1099).
__device__ int mt_continue(AlignState &s, const StepParams &P) {
    if (!s.interval_converged && s.step_iterations < kMaxStepIterations &&
        !(s.psi_t <= 0 && s.d_phi_t <= -kNu * s.d_phi_0)) {
        double a_t;
        if (s.open_interval)
            a_t = trial_value(s.a_l, s.f_l, s.g_l, s.a_u, s.f_u, s.g_u, s.a_t, s.psi_t, s.d_psi_t);
        else
            a_t = trial_value(s.a_l, s.f_l, s.g_l, s.a_u, s.f_u, s.g_u, s.a_t, s.phi_t, s.d_phi_t);
        a_t = std_min(a_t, s.step_max);
        a_t = std_max(a_t, s.step_min);
        s.a_t = a_t;
        for (int i = 0; i < 6; ++i) s.x_t[i] = s.p[i] + s.dir[i] * a_t;
        return kActPose;
    }
    if (s.step_iterations) {  // computeHessian (:1141-1142)
        request(s, P, kEvalHessian, kPhaseMTHess);
        return kActNone;
    }
    return kActEnd;
}

// Consumes the evaluation result held in s.score/g/H (lane 0) up to the next
// thing the warp does.
__device__ int consume(AlignState &s, const StepParams &P) {
    const int phase = s.phase;
    if (phase == kPhaseMTFirst || phase == kPhaseMTIter) {
        s.phi_t = -s.score;
        s.d_phi_t = -(dot6(s.g, s.dir));
        s.psi_t = psi_mt(s.a_t, s.phi_t, s.phi_0, s.d_phi_0, kMu);
        s.d_psi_t = dpsi_mt(s.d_phi_t, s.d_phi_0, kMu);
        if (phase == kPhaseMTIter) {
            if (s.open_interval && (s.psi_t <= 0 && s.d_psi_t >= 0)) {
                s.open_interval = 0;
                s.f_l = s.f_l + s.phi_0 - kMu * s.d_phi_0 * s.a_l;
                s.g_l = s.g_l + kMu * s.d_phi_0;
                s.f_u = s.f_u + s.phi_0 - kMu * s.d_phi_0 * s.a_u;
                s.g_u = s.g_u + kMu * s.d_phi_0;
            }
            bool ic;
            if (s.open_interval)
                ic = update_interval(s.a_l, s.f_l, s.g_l, s.a_u, s.f_u, s.g_u, s.a_t, s.psi_t, s.d_psi_t);
            else
                ic = update_interval(s.a_l, s.f_l, s.g_l, s.a_u, s.f_u, s.g_u, s.a_t, s.phi_t, s.d_phi_t);
            s.interval_converged = ic;
            s.step_iterations++;
        }
        return mt_continue(s, P);
    }
    if (phase == kPhaseMTHess) return kActEnd;
    return phase == kPhaseInitEval ? kActNewton : kActNone;
}

// Advances the alignment until the next evaluation is requested or it is
// done.  Lane 0 runs the state machine; the parts that are long serial chains
// of FP64 operations (the 6x6 solve, the trigonometry) are the warp's: the
// step is bound by the latency of these chains (7.6 -> 5.2 us for one
// alignment, 16.1 -> 10.4 us on average over the rounds of 1024, against all
// of it on lane 0).
__device__ void advance(StepSmem &m, const StepParams &P) {
    const int lane = threadIdx.x & 31;
    AlignState &s = m.st;
    int act = kActNone, first = 0;
    if (lane == 0) {
        act = consume(s, P);
        first = act == kActPose;  // the line search goes on: its gradient at the trial point
    }
    act = bcast0(act);
    first = bcast0(first);
    // bounded: each pass either requests an evaluation, finishes, or
    // completes a Newton iteration without one (d_phi_0 == 0)
    for (int guard = 0; guard <= 1024; ++guard) {
        if (act == kActEnd) {
            if (lane == 0) act = newton_end(s, P) ? kActNone : kActNewton;
            act = bcast0(act);
        }
        if (act == kActNewton) {
            if (guard == 1024) break;
            __syncwarp();
            double dp[6];
            warp_solve6(s.H, s.g, dp);
            if (lane == 0) act = newton_start(s, P, dp);
            act = bcast0(act);
        }
        if (act == kActPose) {
            __syncwarp();
            warp_set_pose(m, P);
            if (lane == 0) {
                if (first)
                    request(s, P, kEvalGradient, kPhaseMTIter);
                else
                    request(s, P, kEvalFull, kPhaseMTFirst);
            }
            return;
        }
        if (act == kActNone) return;
    }
    if (lane == 0) {
        s.status = NDT_ST_WATCHDOG_DEV;
        s.converged = 0;
        s.phase = kPhaseDone;
        s.eval_mode = kEvalNone;
    }
}

// One warp per alignment, on a shared-memory copy of the alignment's state
// (the state machine is serial FP64 code that touches hundreds of fields),
// which the warp moves between global and shared memory in 16-byte pieces.
constexpr int kStateWarps = 4;
constexpr int kAhead = 16;  // chunk partials read at a time
constexpr int kStateVecs = (int)(sizeof(AlignState) / sizeof(uint4));
constexpr int kStatePieces = (kStateVecs + 31) / 32;  // per lane
static_assert(sizeof(AlignState) % sizeof(uint4) == 0, "AlignState is copied in 16-byte pieces");

__device__ __forceinline__ void copy_state(AlignState *dst, const AlignState *src, int lane) {
    const uint4 *s = reinterpret_cast<const uint4 *>(src);
    uint4 *d = reinterpret_cast<uint4 *>(dst);
    for (int i = lane; i < kStateVecs; i += 32) d[i] = s[i];
}

// The state of an alignment before its first evaluation (the whole warp).
__device__ void init_state(StepSmem &m, const float *__restrict__ guess, int n, const StepParams &P) {
    const int lane = threadIdx.x & 31;
    AlignState &s = m.st;
    if (lane < 16) s.T[lane] = guess[lane];
    for (int k = lane; k < 36; k += 32) s.H[k] = 0.0;
    __syncwarp();
    if (lane == 0) {
        pose_vector(P.compat != 0, s.T, s.p);
        for (int i = 0; i < 6; ++i) {
            s.x_t[i] = s.p[i];
            s.dir[i] = 0.0;
            s.g[i] = 0.0;
        }
        s.score = 0.0;
        s.phi_0 = s.d_phi_0 = s.a_l = s.f_l = s.g_l = s.a_u = s.f_u = s.g_u = s.a_t = 0.0;
        s.phi_t = s.d_phi_t = s.psi_t = s.d_psi_t = 0.0;
        s.step_max = P.step_max;
        s.step_min = P.step_min;
        s.nr_iterations = 0;
        s.step_iterations = 0;
        s.open_interval = 1;
        s.interval_converged = 0;
        s.converged = 0;
        s.evals = 0;
        s.status = 0;
        s.n = n;
        s.eval_mode = P.first_mode;
        s.phase = kPhaseInitEval;
    }
    __syncwarp();
    warp_trig(m, s.p);
    if (!P.compat && lane == 1) build_tm_corrected(s.T, s.p, m.c, m.s);
    warp_angles(m, s.p, P.compat != 0);
}

// FP64 sum of the alignment's chunk partials in chunk order (deterministic;
// lane l sums the values l and l + 32, the loads of 16 chunks in flight, the
// state's copy beside them), then the warp advances the state machine; the chunks of an alignment
// that asks for another evaluation go to the active list (their order in it
// changes no result, since each chunk writes its own partial slot).  The last
// block to finish ends the round: the counters that separate launches would
// have to clear or read (four memsets, the list's compaction, the loop
// condition: 10 us of a 21 us round tail) are set here.  A block that is alone
// (up to kStateWarps alignments) keeps them in shared memory: its fences and
// atomics were 1.6 of 7.5 us for one alignment.
__global__ void step_kernel(AlignState *__restrict__ states, const double *__restrict__ partials, TileLists L,
                            double *__restrict__ exc, int B, StepParams P, RoundEnd end) {
    __shared__ StepSmem s_m[kStateWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    RoundCtl *ctl = end.ctl;
    const bool alone = gridDim.x == 1;
    // the round's counters: a single block's own, or all blocks'
    __shared__ unsigned long long s_list;
    __shared__ int s_next;
    unsigned long long *next_list = alone ? &s_list : &ctl->next_list;
    int *next_active = alone ? &s_next : &ctl->next_active;
    int round = 0;
    if (threadIdx.x == 0) {
        s_list = 0ull;
        s_next = 0;
        round = ctl->round_no + 1;
    }
    __syncthreads();
    const int b = blockIdx.x * kStateWarps + warp;
    AlignState *st = states + b;
    int mode = kEvalNone, c0 = 0, c1 = 0;
    if (b < B) {
        mode = st->eval_mode;
        c0 = L.chunk_begin[b];
        c1 = L.chunk_begin[b + 1];
    }
    if (mode != kEvalNone) {
        StepSmem &m = s_m[warp];
        AlignState &s = m.st;
        uint4 piece[kStatePieces];
#pragma unroll
        for (int q = 0; q < kStatePieces; ++q)
            if (lane + 32 * q < kStateVecs) piece[q] = reinterpret_cast<const uint4 *>(st)[lane + 32 * q];
        const bool two = lane + 32 < kPartial;
        double *e = exc + (size_t)b * kPartial + lane;
        const double e0 = e[0], e1 = two ? e[32] : 0.0;
        double v0 = 0.0, v1 = 0.0;
        for (int c = c0; c < c1; c += kAhead) {
            double t0[kAhead], t1[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const double *p = partials + (size_t)(c + u) * kPartial + lane;
                t0[u] = c + u < c1 ? p[0] : 0.0;
                t1[u] = two && c + u < c1 ? p[32] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                if (c + u < c1) {
                    v0 += t0[u];
                    v1 += t1[u];
                }
        }
        m.v[lane] = v0 + e0;
        e[0] = 0.0;
        if (two) {
            m.v[lane + 32] = v1 + e1;
            e[32] = 0.0;
        }
#pragma unroll
        for (int q = 0; q < kStatePieces; ++q)
            if (lane + 32 * q < kStateVecs) reinterpret_cast<uint4 *>(&s)[lane + 32 * q] = piece[q];
        __syncwarp();
        // the evaluation's result (computeDerivatives without a Hessian zeroes it, kernel.cpp:667)
        const bool grad = mode == kEvalFull || mode == kEvalGradient;
        const bool hess = mode == kEvalFull || mode == kEvalHessian;
        if (grad && lane < 6) s.g[lane] = m.v[1 + lane];
        for (int k = lane; k < 36; k += 32) s.H[k] = hess ? m.v[7 + k] : 0.0;
        if (lane == 0) {
            if (grad) s.score = m.v[0];
            s.evals++;
            s.eval_mode = kEvalNone;
        }
        __syncwarp();
        advance(m, P);
        unsigned long long at = 0;
        int nb = 0, ns = 0, b0 = 0, s0 = 0;
        if (lane == 0) {
            if (s.eval_mode != kEvalNone) {
                atomicAdd(next_active, 1);
                if (L.active_chunks) {
                    b0 = L.big_begin[b];
                    nb = L.big_begin[b + 1] - b0;
                    s0 = L.small_begin[b];
                    ns = L.small_begin[b + 1] - s0;
                    at = atomicAdd(next_list, (unsigned long long)nb << 32 | (unsigned)ns);
                }
            }
            atomicAdd(&ctl->counters.evaluations, 1ull);
        }
        __syncwarp();
        copy_state(st, &s, lane);
        if (L.active_chunks) {
            at = __shfl_sync(0xffffffffu, at, 0);
            nb = __shfl_sync(0xffffffffu, nb, 0);
            ns = __shfl_sync(0xffffffffu, ns, 0);
            b0 = __shfl_sync(0xffffffffu, b0, 0);
            s0 = __shfl_sync(0xffffffffu, s0, 0);
            const int at_big = (int)(at >> 32), at_small = (int)(at & 0xffffffffu);
            const int total_big = *L.num_big;
            for (int j = lane; j < nb; j += 32) L.active_chunks[at_big + j] = b0 + j;
            for (int j = lane; j < ns; j += 32) L.active_chunks[L.capacity - 1 - (at_small + j)] = total_big + s0 + j;
        }
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    int active = s_next;
    unsigned long long list = s_list;
    if (!alone) {
        __threadfence();
        if (atomicAdd(&ctl->ticket, 1) != (int)gridDim.x - 1) return;
        __threadfence();
        active = atomicExch(&ctl->next_active, 0);
        list = atomicExch(&ctl->next_list, 0ull);
        ctl->ticket = 0;
    }
    ctl->active = active;
    ctl->num_active[0] = (int)(list >> 32);
    ctl->num_active[1] = (int)(list & 0xffffffffu);
    ctl->work_counter = 0;
    ctl->flag_n = 0;
    atomicAdd(&ctl->counters.rounds, 1ull);
    ctl->round_no = round;
    if (end.graph) {
        // another round while an alignment asked for an evaluation and the round
        // budget (the evaluation watchdog) is not spent, so the loop always ends
        atomicAdd(end.launches, (unsigned long long)end.per_round);
        cudaGraphSetConditional(end.loop, (active > 0 && round < end.max_rounds) ? 1u : 0u);
    }
}

__global__ void finalize_kernel(const AlignState *__restrict__ states, int B, float *__restrict__ out,
                                int *__restrict__ conv, double *__restrict__ fit, int *__restrict__ status,
                                const int *__restrict__ overflow) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= B) return;
    const AlignState &s = states[b];
    for (int k = 0; k < 16; ++k) out[16 * (size_t)b + k] = s.T[k];
    conv[b] = s.converged;
    fit[b] = s.n > 0 ? s.score / (double)s.n : 0.0;
    int st = s.status;
    if (s.phase != kPhaseDone && st == 0) st = NDT_ST_WATCHDOG_DEV;
    if (overflow && *overflow) st |= NDT_ST_OVERFLOW_DEV;
    if (status) status[b] = st;
}

// Chunk plan of an alignment with t tiles: large chunks of kb tiles over the
// first tiles, leaving at least 4 small chunks' worth (4 ks tiles, or all of
// them when t is smaller) for small chunks of ks tiles.
__device__ __forceinline__ void chunk_plan(int t, int kb, int ks, int &nb, int &ns) {
    const int keep = min(t, 4 * ks);
    nb = (t - keep) / kb;
    const int rest = t - nb * kb;
    ns = (rest + ks - 1) / ks;
}

// The scan that alignment b reads (TileLists::scans).
__device__ __forceinline__ int scan_of(const TileLists &L, int b) { return L.scans > 0 ? b % L.scans : b; }

// Tile list: ceil(n_b / tile) tiles per alignment, in alignment order; the
// large and small chunk counts per alignment.
__global__ void tile_count_kernel(const int *__restrict__ offsets, int B, int tile, int kb, int ks, TileLists L) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > B) return;
    if (b == B) {
        L.tile_begin[B] = 0;
        L.big_begin[B] = 0;
        L.small_begin[B] = 0;
        return;
    }
    const int sb = scan_of(L, b);
    const int n = offsets[sb + 1] - offsets[sb];
    const int t = n > 0 ? (n + tile - 1) / tile : 0;
    int nb, ns;
    chunk_plan(t, kb, ks, nb, ns);
    L.tile_begin[b] = t;
    L.big_begin[b] = nb;
    L.small_begin[b] = ns;
}

// Exclusive scans in place of three arrays of n ints, one block of 1024
// threads per array (block k scans arrays[k], total to *totals[k]).
struct ScanArgs {
    int *data[3];
    int *total[3];
};

__global__ void scan3_kernel(ScanArgs a, int n) {
    __shared__ int s_warp[32];
    int *data = a.data[blockIdx.x];
    int *total = a.total[blockIdx.x];
    const int t = threadIdx.x, nt = blockDim.x;
    const int chunk = (n + nt - 1) / nt;
    const int lo = min(n, t * chunk), hi = min(n, lo + chunk);
    int sum = 0;
    for (int i = lo; i < hi; ++i) sum += data[i];
    int lane = t & 31, w = t >> 5;
    int incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
        int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s_warp[w] = incl;
    __syncthreads();
    if (w == 0) {
        int v = (lane < (nt >> 5)) ? s_warp[lane] : 0;
        int inc2 = v;
        for (int o = 1; o < 32; o <<= 1) {
            int u = __shfl_up_sync(0xffffffffu, inc2, o);
            if (lane >= o) inc2 += u;
        }
        s_warp[lane] = inc2 - v;
    }
    __syncthreads();
    int run = s_warp[w] + incl - sum;
    for (int i = lo; i < hi; ++i) {
        int v = data[i];
        data[i] = run;
        run += v;
    }
    if (total && t == nt - 1) *total = run;
}

// One warp writes its alignment's tiles, its chunks (large ones at the front
// of the list, small ones after every large one), its slot range and its
// entries of the first pass's active list.
__device__ __forceinline__ void fill_lists(const int *__restrict__ offsets, int b, int B, int tile, int kb, int ks,
                                           const TileLists &L) {
    const int lane = threadIdx.x & 31;
    const int sb = scan_of(L, b);
    const int lo = offsets[sb], hi = offsets[sb + 1];
    const int t0 = L.tile_begin[b], t1 = L.tile_begin[b + 1];
    for (int t = t0 + lane; t < t1; t += 32) {
        Tile x;
        x.align = b;
        x.start = lo + (t - t0) * tile;
        x.end = min(hi, x.start + tile);
        x.slot = t;
        L.tiles[t] = x;
    }
    const int b0 = L.big_begin[b], nb = L.big_begin[b + 1] - b0;
    const int s0 = L.small_begin[b], ns = L.small_begin[b + 1] - s0;
    const int slot0 = b0 + s0;
    const int total_big = *L.num_big;
    if (lane == 0) {
        L.chunk_begin[b] = slot0;
        if (b == B - 1) L.chunk_begin[B] = *L.num_chunks = slot0 + nb + ns;
    }
    for (int j = lane; j < nb + ns; j += 32) {
        Chunk x;
        x.align = b;
        int pos;
        if (j < nb) {
            x.first = t0 + j * kb;
            x.end = x.first + kb;
            pos = b0 + j;
        } else {
            x.first = t0 + nb * kb + (j - nb) * ks;
            x.end = min(t1, x.first + ks);
            pos = total_big + s0 + (j - nb);
        }
        x.slot = slot0 + j;
        L.chunks[pos] = x;
        if (L.active_chunks) L.active_chunks[j < nb ? pos : L.capacity - 1 - (s0 + j - nb)] = pos;
    }
}

__global__ void tile_fill_kernel(const int *__restrict__ offsets, int B, int tile, int kb, int ks, TileLists L) {
    const int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (b < B) fill_lists(offsets, b, B, tile, kb, ks, L);
}

// Start of a batch, one warp per alignment: its lists and its state.  Thread
// 0 also sets the first pass's active-list counts.
__global__ void fill_init_kernel(const int *__restrict__ offsets, int B, int tile, int kb, int ks, TileLists L,
                                 AlignState *__restrict__ states, const float *__restrict__ guesses, StepParams P,
                                 double *__restrict__ exc, RoundCtl *__restrict__ ctl) {
    __shared__ StepSmem s_m[kStateWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int b = blockIdx.x * kStateWarps + warp;
    if (b >= B) return;
    if (b == 0 && lane == 0) {
        ctl->num_active[0] = *L.num_big;
        ctl->num_active[1] = L.small_begin[B];
    }
    for (int k = lane; k < kPartial; k += 32) exc[(size_t)b * kPartial + k] = 0.0;
    const int sb = scan_of(L, b);
    init_state(s_m[warp], guesses + 16 * (size_t)b, offsets[sb + 1] - offsets[sb], P);
    fill_lists(offsets, b, B, tile, kb, ks, L);
    __syncwarp();
    copy_state(states + b, &s_m[warp].st, lane);
}

// Tile and chunk counts per alignment and their exclusive scans by one block
// (up to kOneBlockLists alignments: three launches in one), and the round
// control cleared.
__device__ __forceinline__ void clear_ctl(RoundCtl *ctl, int reset_counters, int t) {
    static_assert(sizeof(RoundCtl) % 4 == 0 && sizeof(Counters) % 8 == 0, "cleared by words");
    const int head = (int)((sizeof(RoundCtl) - sizeof(Counters)) / 4), all = (int)(sizeof(RoundCtl) / 4);
    if (t < (reset_counters ? all : head)) reinterpret_cast<int *>(ctl)[t] = 0;
}

__global__ void clear_ctl_kernel(RoundCtl *ctl, int reset_counters) { clear_ctl(ctl, reset_counters, threadIdx.x); }

__global__ void __launch_bounds__(1024) lists_kernel(const int *__restrict__ offsets, int B, int tile, int kb, int ks,
                                                     TileLists L, RoundCtl *ctl, int reset_counters) {
    __shared__ int s_warp[3][32];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    clear_ctl(ctl, reset_counters, t);
    const int per = (B + 1023) / 1024;
    const int lo = min(B, t * per), hi = min(B, lo + per);
    int sum[3] = {0, 0, 0};
    for (int b = lo; b < hi; ++b) {
        const int sb = scan_of(L, b);
        const int n = offsets[sb + 1] - offsets[sb];
        const int tiles = n > 0 ? (n + tile - 1) / tile : 0;
        int nb, ns;
        chunk_plan(tiles, kb, ks, nb, ns);
        sum[0] += tiles;
        sum[1] += nb;
        sum[2] += ns;
    }
    int incl[3] = {sum[0], sum[1], sum[2]};
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const int v = __shfl_up_sync(0xffffffffu, incl[q], o);
            if (lane >= o) incl[q] += v;
        }
    if (lane == 31)
        for (int q = 0; q < 3; ++q) s_warp[q][w] = incl[q];
    __syncthreads();
    if (w < 3) {
        const int v = s_warp[w][lane];
        int inc2 = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, inc2, o);
            if (lane >= o) inc2 += u;
        }
        s_warp[w][lane] = inc2 - v;
    }
    __syncthreads();
    int run[3];
    for (int q = 0; q < 3; ++q) run[q] = s_warp[q][w] + incl[q] - sum[q];
    for (int b = lo; b < hi; ++b) {
        L.tile_begin[b] = run[0];
        L.big_begin[b] = run[1];
        L.small_begin[b] = run[2];
        const int sb = scan_of(L, b);
        const int n = offsets[sb + 1] - offsets[sb];
        const int tiles = n > 0 ? (n + tile - 1) / tile : 0;
        int nb, ns;
        chunk_plan(tiles, kb, ks, nb, ns);
        run[0] += tiles;
        run[1] += nb;
        run[2] += ns;
    }
    if (t == 1023) {  // (its run ends at B)
        L.tile_begin[B] = *L.num_tiles = run[0];
        L.big_begin[B] = *L.num_big = run[1];
        L.small_begin[B] = run[2];
    }
}

// One evaluation request at pose p (test hook: the caller supplies the
// transformed points, so T is the identity).
__global__ void prepare_eval_kernel(AlignState *__restrict__ s, const double *__restrict__ p6, int n,
                                    double *__restrict__ exc, int compat) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    for (int k = 0; k < 16; ++k) s->T[k] = (k % 5 == 0) ? 1.0f : 0.0f;
    for (int i = 0; i < 6; ++i) s->x_t[i] = s->p[i] = p6[i];
    double a[kAngle];
    angle_terms(p6, a, compat != 0);
    for (int k = 0; k < kAngle; ++k) {
        s->angd[k] = a[k];
        s->angf[k] = (float)a[k];
    }
    s->n = n;
    s->eval_mode = kEvalFull;
    s->phase = kPhaseInitEval;
    for (int k = 0; k < kPartial; ++k) exc[k] = 0.0;
}

}  // namespace

int launch_prepare_eval(AlignState *d_state, const double *d_p6, int n, double *d_exc, int compat, cudaStream_t st) {
    prepare_eval_kernel<<<1, 32, 0, st>>>(d_state, d_p6, n, d_exc, compat);
    return (int)cudaGetLastError();
}

static void launch_scans(const int *d_offsets, int B, int tile, int kb, int ks, const TileLists &L, cudaStream_t st) {
    tile_count_kernel<<<(B + 1 + 255) / 256, 256, 0, st>>>(d_offsets, B, tile, kb, ks, L);
    ScanArgs a;
    a.data[0] = L.tile_begin;
    a.total[0] = L.num_tiles;
    a.data[1] = L.big_begin;
    a.total[1] = L.num_big;
    a.data[2] = L.small_begin;
    a.total[2] = nullptr;
    scan3_kernel<<<3, 1024, 0, st>>>(a, B + 1);
}

int launch_tiles(const int *d_offsets, int B, int tile, int kb, int ks, const TileLists &L, cudaStream_t st) {
    launch_scans(d_offsets, B, tile, kb, ks, L, st);
    tile_fill_kernel<<<(B * 32 + 255) / 256, 256, 0, st>>>(d_offsets, B, tile, kb, ks, L);
    return (int)cudaGetLastError();
}

int launch_prologue(const int *d_offsets, int B, int tile, int kb, int ks, const TileLists &L, AlignState *d_states,
                    const float *d_guesses, const StepParams &P, double *d_exc, RoundCtl *d_ctl, bool reset_counters,
                    cudaStream_t st, int *launches) {
    if (B <= kOneBlockLists) {
        lists_kernel<<<1, 1024, 0, st>>>(d_offsets, B, tile, kb, ks, L, d_ctl, reset_counters ? 1 : 0);
    } else {
        clear_ctl_kernel<<<1, 64, 0, st>>>(d_ctl, reset_counters ? 1 : 0);
        launch_scans(d_offsets, B, tile, kb, ks, L, st);
    }
    fill_init_kernel<<<(B + kStateWarps - 1) / kStateWarps, 32 * kStateWarps, 0, st>>>(
        d_offsets, B, tile, kb, ks, L, d_states, d_guesses, P, d_exc, d_ctl);
    *launches = prologue_launches(B);
    return (int)cudaGetLastError();
}

int launch_step(AlignState *d_states, const double *d_partials, const TileLists &L, double *d_exc, int B,
                const StepParams &P, const RoundEnd &end, cudaStream_t st) {
    step_kernel<<<(B + kStateWarps - 1) / kStateWarps, 32 * kStateWarps, 0, st>>>(d_states, d_partials, L, d_exc, B,
                                                                                  P, end);
    return (int)cudaGetLastError();
}

// score[b] = the alignment's NDT score (sum over its chunk partials in chunk
// order, plus its FP64 side sum) after one derivative pass.
__global__ void score_kernel(const double *__restrict__ partials, const int *__restrict__ chunk_begin,
                             const double *__restrict__ exc, int B, double *__restrict__ score) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= B) return;
    double v = 0.0;
    for (int c = chunk_begin[b]; c < chunk_begin[b + 1]; ++c) v += partials[(size_t)c * kPartial];
    score[b] = v + exc[(size_t)b * kPartial];
}

int launch_score(const double *d_partials, const int *d_chunk_begin, const double *d_exc, int B, double *d_score,
                 cudaStream_t st) {
    score_kernel<<<(B + 127) / 128, 128, 0, st>>>(d_partials, d_chunk_begin, d_exc, B, d_score);
    return (int)cudaGetLastError();
}

int launch_finalize(const AlignState *d_states, int B, float *d_out, int *d_conv, double *d_fit, int *d_status,
                    const int *d_overflow, cudaStream_t st) {
    finalize_kernel<<<(B + 127) / 128, 128, 0, st>>>(d_states, B, d_out, d_conv, d_fit, d_status, d_overflow);
    return (int)cudaGetLastError();
}

}  // namespace ndt
