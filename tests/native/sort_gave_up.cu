// The radix sort (csrc/grid_build.cu) with waits that give up before their
// first poll: the tiles that wait write nothing, no later tile or pass works on
// what is left (its positions would leave the buffers), and there are no
// segments; the next sort on the same scratch is right again.  Prints "ok" or
// what is wrong.
#include "grid_build.cu"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <numeric>
#include <random>
#include <vector>

int main(int argc, char **argv) {
    const int n = argc > 1 ? std::atoi(argv[1]) : 100000, bits = argc > 2 ? std::atoi(argv[2]) : 22;
    std::mt19937 rng(n + bits);
    std::vector<uint32_t> keys(n);
    for (uint32_t &k : keys) k = rng() & ((1u << bits) - 1u);
    void *scratch = nullptr;
    int32_t *seg_start = nullptr;
    uint32_t *seg_key = nullptr;
    cudaMalloc(&scratch, ndt::sort_scratch_bytes(n));
    cudaMalloc((void **)&seg_start, sizeof(int32_t) * n);
    cudaMalloc((void **)&seg_key, sizeof(uint32_t) * n);
    if (ndt::prepare_sort() != 0) return std::printf("prepare_sort\n"), 1;
    const char *wrong = nullptr;
    auto check = [&](bool ok, const char *what) {
        if (!ok && !wrong) wrong = what;
    };
    for (int turn = 0; turn < 3; ++turn) {
        const bool gives_up = turn == 1;
        ndt::SortBuffers b = ndt::sort_buffers(scratch, n);
        if (gives_up) b.polls = 0;
        uint32_t *in = b.k0, *other = b.k1;
        cudaMemcpy(in, keys.data(), sizeof(uint32_t) * n, cudaMemcpyHostToDevice);
        cudaMemset(other, 0xee, sizeof(uint32_t) * n);
        ndt::sort_segments(b, n, bits, seg_start, seg_key, 0, true);
        check(cudaDeviceSynchronize() == cudaSuccess, "launch");
        int err = -1, nseg = -1;
        cudaMemcpy(&err, ndt::sort_error(b, n), sizeof(int), cudaMemcpyDeviceToHost);
        cudaMemcpy(&nseg, b.nseg, sizeof(int), cudaMemcpyDeviceToHost);
        std::vector<uint32_t> got(n), order(n);
        if (gives_up) {
            check(err == 1 && nseg == 0, "not reported");
            cudaMemcpy(got.data(), in, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost);
            check(got == keys, "a later pass wrote");
            // the first pass: its first tile's pairs at most
            cudaMemcpy(got.data(), other, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost);
            const long long left = std::count(got.begin(), got.end(), 0xeeeeeeeeu);
            check(left >= n - ndt::kSortThreads * ndt::sort_items(n), "a tile that gave up wrote");
            continue;
        }
        check(err == 0, "a healthy sort gave up");
        cudaMemcpy(got.data(), b.k0, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost);
        cudaMemcpy(order.data(), b.v0, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost);
        std::vector<uint32_t> want(n);
        std::iota(want.begin(), want.end(), 0u);
        std::stable_sort(want.begin(), want.end(), [&](uint32_t x, uint32_t y) { return keys[x] < keys[y]; });
        int segs = 0;
        for (int i = 0; i < n; ++i) segs += i == 0 || keys[want[i]] != keys[want[i - 1]];
        bool same = order == want;
        for (int i = 0; i < n; ++i) same = same && got[i] == keys[want[i]];
        check(same && nseg == segs, "sort");
    }
    std::printf("%s\n", wrong ? wrong : "ok");
    return wrong != nullptr;
}
