// label_kernel (csrc/ec.cu) on the states that the racing stores of the pass
// before may leave: any node's parent may be an older ancestor instead of the
// root.  Trees whose nodes hang under random ancestors, least point known at the
// roots only; prints the number of labels that are not their tree's least point.
#include "ec.cu"

#include <cstdio>
#include <cstdlib>
#include <random>

int main(int argc, char **argv) {
    const int n = argc > 1 ? std::atoi(argv[1]) : 1000;
    std::mt19937 rng(n);
    std::vector<int> parent(n), root(n), least(n, 0x7fffffff);
    std::vector<uint32_t> order(n), label(n);
    for (int t = 0; t < n; ++t) {
        order[t] = (uint32_t)t;
        parent[t] = t < 3 || rng() % 50 == 0 ? t : (int)(rng() % t);
        root[t] = parent[t] == t ? t : root[parent[t]];
    }
    std::shuffle(order.begin(), order.end(), rng);
    for (int t = 0; t < n; ++t) least[root[t]] = std::min(least[root[t]], (int)order[t]);
    int *d_parent, *d_least, *d_misc;
    uint32_t *d_order, *d_label;
    for (void **p : {(void **)&d_parent, (void **)&d_least, (void **)&d_order, (void **)&d_label})
        cudaMalloc(p, sizeof(int) * n);
    cudaMalloc((void **)&d_misc, sizeof(int) * 4);
    const int misc[4] = {1, 0, 0, 0};  // segments, the sort's error, status (2)
    cudaMemcpy(d_misc, misc, sizeof(misc), cudaMemcpyHostToDevice);
    cudaMemcpy(d_parent, parent.data(), sizeof(int) * n, cudaMemcpyHostToDevice);
    cudaMemcpy(d_least, least.data(), sizeof(int) * n, cudaMemcpyHostToDevice);
    cudaMemcpy(d_order, order.data(), sizeof(int) * n, cudaMemcpyHostToDevice);
    ec::label_kernel<<<(n + 255) / 256, 256>>>(d_parent, d_order, n, d_misc, d_least, d_misc + 1, d_label, d_misc + 2);
    cudaMemcpy(label.data(), d_label, sizeof(int) * n, cudaMemcpyDeviceToHost);
    int status[2] = {0, 0}, bad = 0;
    cudaMemcpy(status, d_misc + 2, sizeof(status), cudaMemcpyDeviceToHost);
    if (cudaGetLastError() != cudaSuccess || status[1]) return 1;
    for (int t = 0; t < n; ++t) bad += label[order[t]] != (uint32_t)least[root[t]];
    std::printf("%d\n", bad);
    return 0;
}
