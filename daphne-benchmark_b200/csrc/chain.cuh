// Prefix sums chained over the tiles of a launch.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ndt {

// Chained prefixes: tile t of a launch publishes its own sum, then the sum of
// all tiles up to it; a later tile walks back over the published values.
// Tiles are numbered by an atomic ticket, so every tile that one waits for is
// already running and never waits for a later one.  A word holds the state in
// its two top bits and the count below them.
template <class S>
struct Chain {
    static constexpr int kShift = 8 * (int)sizeof(S) - 2;
    static constexpr S kMask = ((S)1 << kShift) - 1;
    static __device__ __forceinline__ void publish(S *w, int flag, S count) {
        *(volatile S *)w = ((S)flag << kShift) | count;
    }
    static __device__ __forceinline__ S load(const S *w) { return *(const volatile S *)w; }
};
constexpr int kOwnSum = 1, kUpToSum = 2;
constexpr int kLookback = 16;                   // words read at a time
constexpr unsigned kChainPolls = 1u << 24;      // polls before a wait gives up (no healthy launch comes near)

// Sum of the counts of the tiles before `tile` in column `col` of state
// [tiles][cols]; *bad = true when a wait gave up (after `limit` polls; 0: before
// the first).
template <class S>
__device__ __forceinline__ S chain_before(const S *state, int tile, int cols, int col, unsigned limit, bool &bad) {
    S sum = 0;
    unsigned polls = 0;
    if (limit == 0) {
        bad = true;
        return 0;
    }
    for (int p = tile - 1; p >= 0;) {
        S v[kLookback];
#pragma unroll
        for (int u = 0; u < kLookback; ++u)
            v[u] = p - u >= 0 ? Chain<S>::load(state + (size_t)(p - u) * cols + col)
                              : (S)kUpToSum << Chain<S>::kShift;
        int used = 0;
        bool end = false, wait = false;
#pragma unroll
        for (int u = 0; u < kLookback; ++u) {
            if (end || wait) continue;
            const int flag = (int)(v[u] >> Chain<S>::kShift);
            if (flag == 0) {
                wait = true;
                continue;
            }
            sum += v[u] & Chain<S>::kMask;
            ++used;
            end = flag == kUpToSum;
        }
        if (end) break;
        p -= used;
        if (wait) {
            if (++polls > limit) {
                bad = true;
                break;
            }
            __nanosleep(100);
        }
    }
    return sum;
}

// The same for one column by a whole warp, 32 words at a time.
__device__ __forceinline__ uint64_t warp_chain_before(const uint64_t *state, int tile, bool &bad) {
    using C = Chain<uint64_t>;
    const int lane = threadIdx.x & 31;
    uint64_t sum = 0;
    unsigned polls = 0;
    for (int p = tile - 1; p >= 0;) {
        const uint64_t v = p - lane >= 0 ? C::load(state + p - lane) : (uint64_t)kUpToSum << C::kShift;
        const int flag = (int)(v >> C::kShift);
        const unsigned ready = __ballot_sync(0xffffffffu, flag != 0), end = __ballot_sync(0xffffffffu, flag == kUpToSum);
        const int run = ready == 0xffffffffu ? 32 : __ffs(~ready) - 1;  // words published without a gap
        const int last = end ? __ffs(end) - 1 : 32;
        const int take = last < run ? last + 1 : run;
        uint64_t mine = lane < take ? v & C::kMask : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
        sum += mine;
        if (last < run) break;
        p -= take;
        if (take < 32 && ++polls > kChainPolls) {
            bad = true;
            break;
        }
    }
    return sum;
}

}  // namespace ndt
