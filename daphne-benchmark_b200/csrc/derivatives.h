// Derivative pass launcher (see derivatives.cu).
#pragma once
#include <cuda_runtime.h>

#include "ndt_types.h"

namespace ndt {

struct EvalArgs {  // (GridDev is in ndt_types.h)
    GridDev grid;
    const float4 *points;  // all scans, concatenated (original coordinates)
    const float4 *trans;   // optional: already transformed points (then T is not applied)
    const Tile *tiles;
    const int *num_tiles;  // device: number of tiles
    const Chunk *chunks;   // chunks of tiles (FP32 pass; the FP64 pass uses chunks of 1 tile)
    const int *num_chunks; // device: number of chunks
    int max_tiles;         // host-side upper bound (grid sizing)
    int tile_size;         // points per tile (must equal the kernel variant's block size)
    AlignState *states;
    double *partials;      // [chunk][kPartial]
    double *exc;           // [alignment][kPartial] FP64 side sums of flagged voxels (FP32 path)
    double d1, d2;         // Gauss constants (kernel.cpp:1181-1185)
    int compat;
    Counters *counters;    // may be null
    int4 *flag_q;          // FP32 path: queue of pairs with flagged voxels (align, point, slot, -)
    unsigned *flag_n;      // queue length (reset by launch_derivatives)
    unsigned flag_cap;     // queue capacity
    int *flag_overflow;    // set when the queue overflowed
    int *work_counter;     // FP32 pass: next chunk (reset by launch_derivatives)
    // FP32 pass, optional: the chunks of the alignments that ask for an
    // evaluation (batches whose alignments finish at different rounds), listed
    // by the step kernel; null: every chunk is handed out and inactive ones
    // skipped.  num_active: large and small chunks in the list.
    int *active_chunks = nullptr;
    const int *num_active = nullptr;
    int active_capacity = 0;
    bool reset = true;     // launch_derivatives clears flag_n and work_counter (else the caller has)
    // FP32 pass: with at most wide_chunks chunks to evaluate, the wide kernel
    // takes them (derivatives_wide.cu; 0: never), which needs the lane sums of
    // its columns (kWideFloats per column of wide_chunks chunks) and a
    // counter per chunk (zero between passes).  expected_chunks: how many a pass
    // has as far as the host can tell (0: no idea), from a bound of the points
    // that the scans need not fill; it saves a launch and decides no result.
    int wide_chunks = 0;
    int expected_chunks = 0;
    float *lane_sums = nullptr;
    unsigned long long *split_state = nullptr;
};

constexpr int kWideFloats = 37 * 32;  // 37 FP32 sums of 32 lanes
constexpr int kWideResident = 3;      // blocks of the wide kernel per SM
constexpr int kWideWaves = 5;
// Chunks up to which the wide kernel is taken: kWideWaves columns per resident
// block (555 chunks of 128-point tiles on 148 SMs).  A wave of it takes 10-15
// us, a pass of the other kernel at least 46 us (one chunk, any number of
// chunks up to 888); with many waves it loses, since its block barriers leave
// issue slots idle (c5-scale batches: 73 ms against 45 ms).  Measured limits of
// 1 / 2 / 3 / 5 / 9 waves, 256 learned-init alignments: 11.20 / 11.09 / 10.93 /
// 10.86 / 11.07 ms.
inline int wide_chunk_limit(int sms, int tile) { return kWideWaves * kWideResident * sms / (tile / 32); }
int prepare_derivatives_wide();
void launch_derivatives_wide(const EvalArgs &args, int sms, cudaStream_t st);

constexpr int kOwn = 27;        // accepted pairs of one point per collect call, at most (3 x 3 x 3 probes)
constexpr int kChunkBig = 8;    // tiles per large chunk of the FP32 pass by default (the FP64 pass: 1)
constexpr int kMaxChunkTiles = 64;
// the chunk sizes the autotuner times (8 suits batches of many large scans,
// c5: 21k chunks per pass; 4 the smaller c3 / c4 batches, where the end of
// the pass is a larger share)
constexpr int kChunkChoices[] = {4, 6, 8};
constexpr int kChunkSmall = 4;  // tiles per small chunk of the FP32 pass, at most the large size (the FP64 pass: 1)

// Per-device set-up (dynamic shared memory opt-in); call with the device current.
int prepare_derivatives();

// FP32 derivative-pass launch shapes the autotuner chooses from:
// (points per tile = threads per block, resident blocks per SM).
struct DerivVariant {
    int tile;
    int min_blocks;
};
constexpr int kNumDerivVariants = 7;
// The shape a new context starts with: 128 threads x 6 blocks per SM (80
// registers, 35.7 KB of shared memory per block), the fastest on B200 for the
// corrected-mode workloads (c5: 2M-point map at 0.5 m); on c2 compat 128 x 5
// is within 1 %.
constexpr int kDefaultDerivVariant = 6;
extern const DerivVariant kDerivVariants[kNumDerivVariants];

// precision 0 = FP32 pair arithmetic (launch shape `variant`), 1 = FP64
// (256-point tiles).  The persistent grid is sms x resident blocks; blocks
// loop over the tiles.
int launch_derivatives(const EvalArgs &args, int precision, int variant, int sms, cudaStream_t st);
// The FP64 pass alone (256-point tiles).
int launch_derivatives_f64(const EvalArgs &args, int sms, cudaStream_t st);
// Kernel launches of one launch_derivatives call (FP32: one or both kernels of
// the pass, and the flagged pairs; FP64: the pass).  Where the wide kernel is
// not launched (its empty launch is about 2 us a round), the other one takes
// every pass, whatever its number of chunks; where both are, the number on the
// device says which of them returns at once.
inline bool launches_wide(const EvalArgs &a) { return a.wide_chunks > 0 && a.expected_chunks <= a.wide_chunks; }
inline bool launches_many(const EvalArgs &a) { return !launches_wide(a) || a.max_tiles > a.wide_chunks; }
inline int derivative_launches(const EvalArgs &a, int precision) {
    return precision == 1 ? 1 : 1 + (launches_wide(a) ? 1 : 0) + (launches_many(a) ? 1 : 0);
}

}  // namespace ndt
