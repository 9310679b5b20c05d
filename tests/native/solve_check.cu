// warp_solve6 (csrc/warp_solve.cuh) against solve6 (csrc/ndt_math.cuh, pinned
// to the reference's solve by test_ndt_math_host.py): the same bits on N
// seeded systems of one kind.  Prints the number of entries that differ.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "ndt_math.cuh"
#include "warp_solve.cuh"

__global__ void solve_kernel(const double *H, const double *g, double *xw, double *xs) {
    const int b = blockIdx.x, lane = threadIdx.x;
    __shared__ double sH[36], sg[6];
    if (lane < 6) sg[lane] = g[6 * b + lane];
    for (int k = lane; k < 36; k += 32) sH[k] = H[36 * b + k];
    __syncwarp();
    double x[6];
    ndt::warp_solve6(sH, sg, x);
    if (lane == 0) {
        double A[6][6], r[6], y[6];
        for (int i = 0; i < 6; ++i) {
            r[i] = -sg[i];
            for (int j = 0; j < 6; ++j) A[i][j] = sH[6 * i + j];
        }
        ndt::solve6(y, A, r);
        for (int i = 0; i < 6; ++i) {
            xw[6 * b + i] = x[i];
            xs[6 * b + i] = y[i];
        }
    }
}

int main(int argc, char **argv) {
    const int kind = argc > 1 ? std::atoi(argv[1]) : 0, N = 4000;
    std::vector<double> H(36 * N), g(6 * N), a(6 * N), b(6 * N);
    std::mt19937_64 rng(7 + kind);
    std::uniform_real_distribution<double> u(-50.0, 50.0);
    for (double &v : H) v = u(rng);
    for (double &v : g) v = u(rng);
    for (int n = 0; n < N; ++n) {
        double *h = &H[36 * n];
        for (int i = 0; i < 6; ++i) {
            if (kind == 1)
                for (int j = 0; j < i; ++j) h[6 * i + j] = h[6 * j + i];  // symmetric
            if (kind == 2) h[6 * i + n % 6] = 0.0;                       // a zero column (pivot 0.001)
            if (kind == 3) h[6 * 2 + i] = h[6 * 4 + i];                  // equal rows
            if (kind == 4) h[6 * i + n % 6] = i % 2 ? 3.0 : -3.0;        // equal pivots
        }
        if (kind == 5) h[n % 36] = n % 3 == 0 ? NAN : (n % 3 == 1 ? INFINITY : -INFINITY);
        if (kind == 6) std::memset(h, 0, sizeof(double) * 36);
    }
    double *dH, *dg, *da, *db;
    cudaMalloc(&dH, sizeof(double) * H.size());
    cudaMalloc(&dg, sizeof(double) * g.size());
    cudaMalloc(&da, sizeof(double) * a.size());
    cudaMalloc(&db, sizeof(double) * b.size());
    cudaMemcpy(dH, H.data(), sizeof(double) * H.size(), cudaMemcpyHostToDevice);
    cudaMemcpy(dg, g.data(), sizeof(double) * g.size(), cudaMemcpyHostToDevice);
    solve_kernel<<<N, 32>>>(dH, dg, da, db);
    cudaMemcpy(a.data(), da, sizeof(double) * a.size(), cudaMemcpyDeviceToHost);
    cudaMemcpy(b.data(), db, sizeof(double) * b.size(), cudaMemcpyDeviceToHost);
    if (cudaGetLastError() != cudaSuccess) return 1;
    int bad = 0;
    for (size_t i = 0; i < a.size(); ++i)
        if (std::memcmp(&a[i], &b[i], sizeof(double)) && !(std::isnan(a[i]) && std::isnan(b[i]))) ++bad;
    std::printf("%d\n", bad);
    return 0;
}
