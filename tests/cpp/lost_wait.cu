// Grid reductions whose barrier is never completed: a block that does not take part, and waits that run out
// after a few polls.  Prints, for each form of the sum, whether every total is NaN; then the same sums
// with both blocks taking part.
#include <cmath>
#include <cstdio>
#include "gridred.cuh"

namespace cb {

__global__ void sums(double* slots, double* out, int absent) {
    if ((int)blockIdx.x == absent) return;
    GridRed grid(slots);
    double v[2] = {1., 2.}, t[2], w[2] = {3., 4.}, u[2];
    int parity = 0;
    gr_ordered_sum<2>(grid, w, slots + 16, parity, u);
    grid.sync();
    grid.sum<2>(v, t);
    if (blockIdx.x == 0 && threadIdx.x == 0) { out[0] = u[0]; out[1] = u[1]; out[2] = t[0]; out[3] = t[1]; }
}

}  // namespace cb

int main() {
    const int blocks = 2, threads = 64;
    const size_t doubles = cb::gr_doubles(blocks) + cb::gr_ordered_doubles(blocks);
    double *slots, *out, host[4];
    if (cudaMalloc(&slots, doubles * sizeof(double)) != cudaSuccess || cudaMalloc(&out, sizeof(host)) != cudaSuccess) return 2;
    for (int absent : {1, -1}) {
        cudaMemset(slots, 0, doubles * sizeof(double));
        void* args[3] = {&slots, &out, &absent};
        if (cudaLaunchCooperativeKernel((const void*)cb::sums, dim3(blocks), dim3(threads), args, 0, 0) != cudaSuccess) return 2;
        if (cudaMemcpy(host, out, sizeof(host), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
        if (absent >= 0) std::printf("lost %d %d %d %d\n", std::isnan(host[0]), std::isnan(host[1]), std::isnan(host[2]), std::isnan(host[3]));
        else std::printf("whole %g %g %g %g\n", host[0], host[1], host[2], host[3]);
    }
    return 0;
}
