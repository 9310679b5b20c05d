// The FP32 derivative pass for few chunks (derivatives_f32.cu holds the pass
// for many).
//
// With few chunks the other kernel is bound by one serial chain: a warp takes
// its 32 points of up to 8 tiles one after the other, each a chain of
// dependent gathers (window offsets, entries, pair records) of about 5 us,
// while most SMs have nothing to do.  One 8000-point scan is 11 chunks: 46.6
// us per evaluation on B200.  This kernel gives every tile column a warp of
// its own: 15.2 us for the same bits, 13.1 with one atomic for a column's end
// (its pairs and its count together, after one fence), none for blocks that
// have no second item, and the first tile and point read beside the state.
// Reading the pairs' records ahead into L1 gained nothing.
#include <cuda_runtime.h>
#include <stdint.h>

#include "derivatives.h"
#include "pair_f32.cuh"
#include "probe.cuh"

namespace ndt {

namespace {

// A tile's points fall into columns of 32 (column w = points 32 w .. 32 w + 31);
// a column's lane sums are FP32 chains over the chunk's tiles, whose order is
// part of the result.  Here a block takes one column of a chunk, one warp per
// tile (kStepWarps tiles at a time): the warps search and evaluate at the same
// time, each leaving its step's contributions in shared memory, and the chains
// are then added up in tile order, one (value, lane) per thread, so the sums
// equal the other kernel's bit for bit.  The block that finishes a chunk's
// last column adds the columns up in FP64.
constexpr int kStepWarps = 8;
constexpr int kBlock = 32 * kStepWarps;
// A tile column with more pairs than kDenseThreshold is evaluated per point;
// fewer go to the column's ring of deferred pairs, evaluated 32 at a time.
constexpr int kDenseThreshold = 32;
// ring: what is left of the tiles before (fewer than 32 pairs) and at most
// kDenseThreshold pairs from each warp's tile
constexpr int kRing = 32 + kStepWarps * kDenseThreshold;
static_assert(kOwn <= kAcc, "a warp's pair list lies where its contributions go");

struct WideSmem {
    // per warp: its tile's accepted pairs (own[k][lane], k < kOwn), then its
    // step's contributions (value k of lane l at 32 k + l)
    unsigned step[kStepWarps][kAcc * 32];
    float carry[kAcc][32];   // lane sums of the current column (chunks of more than kStepWarps tiles)
    uint2 ring[kRing];       // deferred pairs: (slot << 6 | flag << 5, point index)
};

// Orders the steps of one group of tiles.  Lane t < kStepWarps describes warp
// t's tile: n pairs; dense (n > kDenseThreshold) tiles are a step of their
// own, the others append to the ring, whose round r (32 pairs) runs after the
// first tile that fills it (`partial`: the last, partial round runs after the
// last tile).  Sparse warp number r executes round r.  Returns the number of
// steps and, in `order`, the executing warps in step order, 4 bits each.
__device__ __forceinline__ int step_order(int n, unsigned incl, int rounds, bool partial, bool flush_only,
                                          unsigned sparse_mask, unsigned &order) {
    const int lane = threadIdx.x & 31;
    const bool dense = n > kDenseThreshold;
    const int r = __popc(sparse_mask & lanemask_lt());
    const bool runs = ((sparse_mask >> lane) & 1u) && r < rounds;
    const unsigned need = 32u * (unsigned)(r + 1);
    int key = 99, after = 0;
    for (int i = 0; i < kStepWarps; ++i) after += __shfl_sync(kFull, incl, i) < need;
    if (lane < kStepWarps) {
        if (dense) key = 2 * lane;
        if (runs) key = (partial && r == rounds - 1) ? 2 * kStepWarps + 1 : 2 * after + 1;
        if (flush_only && lane == 0) key = 0;
    }
    int pos = 0;
    for (int i = 0; i < kStepWarps; ++i) pos += __shfl_sync(kFull, key, i) < key;
    order = __reduce_or_sync(kFull, key < 99 ? (unsigned)lane << (4 * pos) : 0u);
    return __popc(__ballot_sync(kFull, key < 99));
}

// COMPAT: the reference's Hessian form and pose build (else corrected); WIN: the
// map has a probe-window table (the neighbour search compiles only the paths it
// can take, a smaller instruction footprint).  W: columns of a tile.
template <int W, bool COMPAT, bool WIN>
__global__ void __launch_bounds__(kBlock, kWideResident) derivative_wide_kernel(const __grid_constant__ EvalArgs args) {
    __shared__ float s_T[12];
    __shared__ float s_ang[kAngle];
    __shared__ int s_mode;
    __shared__ double s_tot[kAcc];
    __shared__ int s_n[kStepWarps];      // pairs of each warp's tile in the current group
    __shared__ unsigned s_pairs, s_chunk_pairs;  // pairs of the current column, of its chunk
    __shared__ int s_item[2];
    __shared__ int s_more;               // a tile has probes left (see `serial`)
    __shared__ int s_last;
    // work counters (points, tiles, probes, occupied probes, pairs) per warp, kept
    // only when the caller asked for counters (in shared memory: no registers)
    __shared__ unsigned long long s_work[kStepWarps][5];
    extern __shared__ __align__(16) unsigned char s_dyn[];
    WideSmem &sm = *reinterpret_cast<WideSmem *>(s_dyn);

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const GridDev &grid = args.grid;
    unsigned (*own)[32] = reinterpret_cast<unsigned (*)[32]>(sm.step[warp]);
    float *contrib = reinterpret_cast<float *>(sm.step[warp]) + lane;
    const float d1 = (float)args.d1, d2 = (float)args.d2;

    const int nc = pass_chunks(args);
    if (nc > args.wide_chunks) return;  // the other kernel's
    const int items = nc * W;  // (chunk, column)
    if (threadIdx.x == 0) {
        s_more = 0;
        s_pairs = 0;
    }
    if (lane == 0)
        for (int q = 0; q < 5; ++q) s_work[warp][q] = 0;
    int parity = 0;

    // A block's first item is its own index, the others are handed out (one
    // atomic each).  (No block takes more than `items` items; the bound only
    // guards against a corrupted counter.)
    for (int it = 0; it <= items; ++it) {
        if (it > 0 && items <= (int)gridDim.x) break;  // every block had its own
        if (threadIdx.x == 0)
            s_item[parity] = it == 0 ? (int)blockIdx.x : (int)gridDim.x + atomicAdd(args.work_counter, 1);
        __syncthreads();
        const int item = s_item[parity];
        parity ^= 1;
        if (item >= items) break;
        const int slot_k = item / W, w = item % W;
        const Chunk ck = args.chunks[active_chunk(args, slot_k)];
        const AlignState *st = args.states + ck.align;
        // this warp's tile and point of the first group, beside the state
        Tile first_tile = {};
        float4 first_x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ck.first + warp < ck.end) {
            first_tile = args.tiles[ck.first + warp];
            const int i = first_tile.start + 32 * w + lane;
            if (i < first_tile.end) first_x = args.points[i];
        }
        if (threadIdx.x == 0) s_mode = st->eval_mode;
        if (threadIdx.x < 12) s_T[threadIdx.x] = st->T[threadIdx.x];
        if (threadIdx.x < kAngle) s_ang[threadIdx.x] = st->angf[threadIdx.x];
        __syncthreads();
        const int mode = s_mode;
        if (mode == kEvalNone) continue;  // s_mode is rewritten only after the next item's barrier
        const int level = eval_level(mode);
        const int values = level_values(level);
        const int ntiles = ck.end - ck.first;

        // Groups of up to kStepWarps tiles, one warp each.  `serial`: a tile's
        // probes did not fit one collect call (trip counts of 4, coordinates
        // beyond ~1e6 m): from that group on, warp 0 takes the tiles one
        // collect call at a time.
        int g = 0, resume = 0;
        unsigned carried = 0;  // pairs in the ring from earlier groups
        bool serial = false, fresh = true;
        for (;;) {
            const int left = ntiles - g;
            const int nt = serial ? min(1, left) : min(kStepWarps, left);
            const bool mine = warp < nt;
            int c = 0, i = 0;
            bool more = false;
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            float px = 0.f, py = 0.f, pz = 0.f;
            unsigned n_probe = 0, n_occ = 0;
            int n = 0, tile_points = 0;
            if (mine) {
                const Tile tile = g == 0 ? first_tile : args.tiles[ck.first + g + warp];
                i = tile.start + 32 * w + lane;
                const bool valid = i < tile.end;
                tile_points = tile.end - tile.start;
                if (valid) x = g == 0 ? first_x : args.points[i];
                // transformPointCloud (kernel.cpp:397-400), float, left to right
                if (args.trans) {
                    const float4 y = valid ? args.trans[i] : make_float4(0.f, 0.f, 0.f, 0.f);
                    px = y.x; py = y.y; pz = y.z;
                } else {
                    px = transform_row(s_T, x.x, x.y, x.z);
                    py = transform_row(s_T + 4, x.x, x.y, x.z);
                    pz = transform_row(s_T + 8, x.x, x.y, x.z);
                }
                OwnSink sink{own, 0};
                collect_pairs<OwnSink, WIN ? kProbeWindows : kProbeDenseIndex>(grid, px, py, pz, valid, sink,
                                                                               n_probe, n_occ, resume);
                c = sink.c;
                n = __reduce_add_sync(kFull, c);
                more = resume >= 0;
                if (more && lane == 0) s_more = 1;
            }
            if (lane == 0) s_n[warp] = n;
            __syncthreads();
            const bool again = s_more != 0;
            if (again && !serial) {  // this group again, one collect call at a time
                serial = true;
                resume = 0;
                __syncthreads();
                if (threadIdx.x == 0) s_more = 0;
                continue;
            }
            // the ring's positions, rounds and the order of the steps
            const int nl = lane < kStepWarps ? s_n[lane] : 0;
            const bool sp = nl > 0 && nl <= kDenseThreshold;
            const unsigned sparse_mask = __ballot_sync(kFull, sp);
            unsigned order = 0x76543210u;
            int steps = 0, rounds = 0;
            unsigned total = carried;
            bool from_ring = false;
            int r = 0;
            const bool end = !again && g + nt == ntiles;  // the column's last group
            bool done = end;
            if (sparse_mask == 0u && carried == 0u) {  // dense or empty tiles only
                const unsigned dm = __ballot_sync(kFull, nl > 0);
                steps = __popc(dm);
                if (dm != (1u << steps) - 1u)
                    order = __reduce_or_sync(
                        kFull, nl > 0 ? (unsigned)lane << (4 * __popc(dm & lanemask_lt())) : 0u);
            } else {
                unsigned incl = sp ? (unsigned)nl : 0u;
#pragma unroll
                for (int o = 1; o < kStepWarps; o <<= 1) {
                    const unsigned v = __shfl_up_sync(kFull, incl, o);
                    if (lane >= o) incl += v;
                }
                incl += carried;
                total = __shfl_sync(kFull, incl, kStepWarps - 1);
                const int ns = __popc(sparse_mask);
                const bool flush_only = nt == 0;
                rounds = (int)(total >> 5);
                // the partial round: now if a warp is free for it, else in a group of its own
                const bool partial = end && (total & 31u) && (flush_only || rounds < ns);
                done = end && (partial || (total & 31u) == 0u);
                if (partial) ++rounds;
                steps = step_order(nl, incl, rounds, partial, flush_only, sparse_mask, order);
                r = flush_only ? 0 : __popc(sparse_mask & ((1u << warp) - 1u));
                const bool sparse = (sparse_mask >> warp) & 1u;
                from_ring = flush_only ? warp == 0 : (sparse && r < rounds);
                if (sparse) {
                    int pre = c;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int v = __shfl_up_sync(kFull, pre, o);
                        if (lane >= o) pre += v;
                    }
                    pre += (int)__shfl_sync(kFull, incl, warp) - n - c;
                    for (int k = 0; k < c; ++k) sm.ring[pre + k] = make_uint2(own[k][lane] & ~31u, (unsigned)i);
                }
                __syncthreads();  // the ring is complete
            }
            // work counters; the pairs feed the partial's count
            if (mine) {
                if (lane == 0 && n) atomicAdd(&s_pairs, (unsigned)n);
                if (args.counters) {
                    const unsigned probes = __reduce_add_sync(kFull, n_probe);
                    const unsigned occupied = __reduce_add_sync(kFull, n_occ);
                    if (lane == 0) {
                        if (w == 0 && !more) {
                            s_work[warp][0] += (unsigned)tile_points;
                            s_work[warp][1] += 1;
                        }
                        s_work[warp][2] += probes;
                        s_work[warp][3] += occupied;
                        s_work[warp][4] += (unsigned)n;
                    }
                }
            }
            // this warp's step: its tile's points (dense), each lane its own
            // pairs, or round r of the ring, one pair per lane (the lane
            // reloads the pair's point and transforms it again with the same
            // float operations).  Pairs with a flagged voxel are queued for
            // flagged_kernel instead.
            if (n > kDenseThreshold || from_ring) {
                int cnt = c;
                unsigned rcode = 0;
                if (from_ring) {
                    const int at = 32 * r + lane;
                    cnt = at < (int)total ? 1 : 0;
                    if (cnt) {
                        const uint2 d = sm.ring[at];
                        rcode = d.x;
                        i = (int)d.y;
                        x = __ldg(args.points + i);
                        if (args.trans) {
                            const float4 y = __ldg(args.trans + i);
                            px = y.x; py = y.y; pz = y.z;
                        } else {
                            px = transform_row(s_T, x.x, x.y, x.z);
                            py = transform_row(s_T + 4, x.x, x.y, x.z);
                            pz = transform_row(s_T + 8, x.x, x.y, x.z);
                        }
                    }
                }
                PairSums F;
                zero(F);
                const int maxc = __reduce_max_sync(kFull, cnt);
                for (int k = 0; k < maxc; ++k) {
                    if (k < cnt) {
                        const unsigned code = from_ring ? rcode : own[k][lane];
                        const int slot = (int)(code >> 6);
                        if (code & 32u)
                            queue_flagged(args, ck.align, i, slot);
                        else
                            add_pair(grid, F, slot, px, py, pz, d1, d2, level);
                    }
                }
                if (cnt > 0 && !(from_ring && (rcode & 32u)))
                    contract<false>(F, x.x, x.y, x.z, s_ang, contrib, 32, d2, level, COMPAT);
                else
                    for (int k = 0; k < values; ++k) contrib[32 * k] = 0.0f;
            }
            __syncthreads();  // every step's contributions are in place
#pragma unroll 1
            for (int k = warp; k < values; k += kStepWarps) {
                if (!COMPAT && (k == 31 || k == 34 || k == 35)) continue;  // (lower triangle of R: not used)
                float v = fresh ? 0.0f : sm.carry[k][lane];
                for (int q = 0; q < steps; ++q)
                    v += __uint_as_float(sm.step[(order >> (4 * q)) & 15u][32 * k + lane]);
                if (!done)
                    sm.carry[k][lane] = v;
                else
                    __stcg(args.lane_sums + ((size_t)item * kAcc + k) * 32 + lane, v);
            }
            fresh = false;
            if (carried || !done) {  // what the ring keeps for the next group
                if (warp == 0 && (int)total - 32 * rounds > lane) {
                    const uint2 d = sm.ring[32 * rounds + lane];
                    sm.ring[lane] = d;
                }
                if (threadIdx.x == 0) s_more = 0;
            }
            carried = total > 32u * (unsigned)rounds ? total - 32u * (unsigned)rounds : 0u;
            __syncthreads();  // the contributions are read, the ring is moved
            if (done) break;
            if (!again) {
                g += nt;
                resume = 0;
            }
        }
        // the last of the chunk's columns adds them up
        // (the barrier above has the block's lane sums before thread 0's fence)
        if (threadIdx.x == 0) {
            unsigned long long *state = args.split_state + slot_k;  // columns done << 32 | their pairs
            const unsigned long long add = 1ull << 32 | s_pairs;
            s_pairs = 0;
            __threadfence();
            const unsigned long long sum = atomicAdd(state, add) + add;
            s_last = (int)(sum >> 32) == W;
            if (s_last) {
                __threadfence();
                s_chunk_pairs = (unsigned)sum;
                *state = 0ull;
            }
        }
        __syncthreads();
        if (!s_last) continue;
        double *out = args.partials + (size_t)ck.slot * kPartial;
        const unsigned np = s_chunk_pairs;
        if (np == 0) {  // block-uniform; the sums are zero
            if (threadIdx.x < kPartial) out[threadIdx.x] = 0.0;
        } else {
            // the lane sums in FP64 over the columns in order (B200 issues FP64 adds at
            // half the FP32 rate, and the sums of FP32 values stay exact or nearly
            // so), then over the lanes with a fixed shuffle tree
#pragma unroll 1
            for (int k = warp; k < values; k += kStepWarps) {
                double sum = 0.0;
#pragma unroll
                for (int q = 0; q < W; ++q)
                    sum += (double)__ldcg(args.lane_sums + ((size_t)(slot_k * W + q) * kAcc + k) * 32 + lane);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
                if (lane == 0) s_tot[k] = sum;
            }
            __syncthreads();
            if (threadIdx.x < kPartial) {
                const int k = threadIdx.x;
                double v = 0.0;
                if (k < 7) {
                    if (k < values) v = s_tot[k];
                } else if (k == 43) {
                    v = (double)np;
                } else if (values == kAcc) {
                    v = h_entry(s_tot, (k - 7) / 6, (k - 7) % 6, COMPAT ? -args.d2 : 1.0, COMPAT);
                }
                out[k] = v;
            }
        }
    }
    if (args.counters && lane == 0 && (s_work[warp][2] | s_work[warp][1])) {
        if (s_work[warp][1]) {
            atomicAdd(&args.counters->points, s_work[warp][0]);
            atomicAdd(&args.counters->tiles, s_work[warp][1]);
        }
        atomicAdd(&args.counters->probes, s_work[warp][2]);
        atomicAdd(&args.counters->occupied_probes, s_work[warp][3]);
        atomicAdd(&args.counters->pairs, s_work[warp][4]);
    }
}

template <int W>
cudaError_t prepare_one() {
    const int bytes = (int)sizeof(WideSmem);
    const void *k[4] = {(const void *)derivative_wide_kernel<W, true, true>,
                        (const void *)derivative_wide_kernel<W, true, false>,
                        (const void *)derivative_wide_kernel<W, false, true>,
                        (const void *)derivative_wide_kernel<W, false, false>};
    cudaError_t e = cudaSuccess;
    for (const void *f : k) {
        const cudaError_t r = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (r != cudaSuccess) e = r;
    }
    return e;
}

template <int W>
void launch_one(const EvalArgs &args, int sms, cudaStream_t st) {
    const size_t smem = sizeof(WideSmem);
    const long long want = (long long)(args.max_tiles < args.wide_chunks ? args.max_tiles : args.wide_chunks) * W;
    const int blocks = (int)(want < sms * kWideResident ? want : sms * kWideResident);
    const bool win = args.grid.win != nullptr;
    if (args.compat) {
        if (win)
            derivative_wide_kernel<W, true, true><<<blocks, kBlock, smem, st>>>(args);
        else
            derivative_wide_kernel<W, true, false><<<blocks, kBlock, smem, st>>>(args);
    } else {
        if (win)
            derivative_wide_kernel<W, false, true><<<blocks, kBlock, smem, st>>>(args);
        else
            derivative_wide_kernel<W, false, false><<<blocks, kBlock, smem, st>>>(args);
    }
}

}  // namespace

int prepare_derivatives_wide() {
    const cudaError_t a = prepare_one<4>(), b = prepare_one<8>();
    return (int)(a != cudaSuccess ? a : b);
}

void launch_derivatives_wide(const EvalArgs &args, int sms, cudaStream_t st) {
    if (args.tile_size == 256)
        launch_one<8>(args, sms, st);
    else
        launch_one<4>(args, sms, st);
}

}  // namespace ndt
