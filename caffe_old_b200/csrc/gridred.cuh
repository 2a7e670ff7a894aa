// Grid-wide sums for persistent kernels (every block resident: cooperative launch).
//
// A reduction: each warp sums its K values by halving (at each of the first three steps a lane
// keeps half of the values it still holds, 9 shuffles for up to 8 values instead of 5 per value);
// one warp sums the block's warps, stores the block's 8 partials and adds 1 to a counter
// (release); one thread per block polls the counter (acquire); then every block
// sums all blocks' partials in the same order.  Every block gets the same bits.
//
// Measured (us per reduction of 2 / 5 values): 148 blocks of 512 threads 2.4 / 2.7, 296 blocks
// 3.3 / 3.5, 8 blocks 1.5 / 1.7; the former cooperative-groups barrier followed by a read of the
// partials 4.8 on 148 blocks; blocks polling each other's flagged 16-byte partials directly,
// without a counter, 5.3 / 10.4 (lines that many SMs poll are slow to write).
//
// Partials alternate between two buffers: a block can only write reduction n + 2 over n after
// every block has counted into n + 1, that is, after it has read n.  Every wait is bounded: a
// block whose wait ran out takes NaN for the totals of this and every later reduction, and the
// solvers end on a NaN norm.
#pragma once
#include "common.cuh"

namespace cb {

constexpr int GR_VALUES = 16;         // values of one reduction at most
constexpr int GR_THREADS = 1024;      // threads of a block at most; one block per SM at most
#ifndef CAFFE_GR_POLLS
#define CAFFE_GR_POLLS 4000000
#endif
constexpr int GR_POLLS = CAFFE_GR_POLLS;   // polls of the counter before a wait gives up (4 million: seconds)

// doubles of slot memory for a grid of `blocks` blocks: the counter's line, two buffers of partials
inline size_t gr_doubles(int blocks) { return 16 + (size_t)2 * GR_VALUES * blocks; }

// the counter starts at 0: run by the kernel that precedes the reducing one on its stream
__device__ __forceinline__ void gr_clear(double* slots) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *reinterpret_cast<unsigned*>(slots) = 0u;
}

// Warp sums of v[0..K): lane l ends up with the total of value l & 7 (0 for values beyond K).
template <int K>
__device__ __forceinline__ double gr_warp_sums(const double (&v)[K], int lane) {
    double a[4], b[2], c;
    const bool h4 = lane & 4, h2 = lane & 2, h1 = lane & 1;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double lo = i < K ? v[i < K ? i : 0] : 0., hi = i + 4 < K ? v[i + 4 < K ? i + 4 : 0] : 0.;
        a[i] = (h4 ? hi : lo) + __shfl_xor_sync(0xffffffffu, h4 ? lo : hi, 4);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) b[i] = (h2 ? a[i + 2] : a[i]) + __shfl_xor_sync(0xffffffffu, h2 ? a[i] : a[i + 2], 2);
    c = (h1 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, h1 ? b[0] : b[1], 1);
    c += __shfl_xor_sync(0xffffffffu, c, 8);
    c += __shfl_xor_sync(0xffffffffu, c, 16);
    return c;
}

struct GridRed {
    double* slots;
    unsigned n = 0;      // reductions so far
    bool dead = false;   // a wait ran out

    __device__ explicit GridRed(double* s) : slots(s) {}

    // out[q] = sum over every thread of the grid of v[q]
    template <int K>
    __device__ __forceinline__ void sum(const double (&v)[K], double (&out)[K]) {
        static_assert(K <= GR_VALUES, "partials of one reduction");
        __shared__ double sm[GR_THREADS / 32][GR_VALUES];
        __shared__ double st[GR_THREADS / 32][GR_VALUES];
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5, G = gridDim.x;
        ++n;
        double* part = slots + 16 + (size_t)(n & 1u) * GR_VALUES * G;
        constexpr int C = (K + 7) / 8;           // warps sum up to 8 values at a time
        auto warp_sums = [&](const double (&x)[K], double (*dst)[GR_VALUES]) {
#pragma unroll
            for (int h = 0; h < C; ++h) {
                double part8[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) part8[i] = 8 * h + i < K ? x[8 * h + i < K ? 8 * h + i : 0] : 0.;
                const double c = gr_warp_sums(part8, lane);
                if (lane < 8) dst[w][8 * h + lane] = c;
            }
        };
        warp_sums(v, sm);
        __syncthreads();
        int lost = 0;
        if (w == 0) {
#pragma unroll
            for (int h = 0; h < C; ++h) {
                double t = 0.;
                for (int u = lane >> 3; u < nw; u += 4) t += sm[u][8 * h + (lane & 7)];
                t += __shfl_xor_sync(0xffffffffu, t, 8);
                t += __shfl_xor_sync(0xffffffffu, t, 16);
                if (lane < 8 && 8 * h + lane < K) part[(size_t)(8 * h + lane) * G + blockIdx.x] = t;
            }
            __syncwarp();
            // releases this block's writes: the other threads' came before the barrier above
            if (lane == 0) lost = arrive_and_wait();
        }
        if (__syncthreads_or(lost)) dead = true;
        const int ns = min((G + 31) >> 5, nw);   // warps that sum the blocks' partials
        if (w < ns) {
            double t[K];
#pragma unroll
            for (int q = 0; q < K; ++q) t[q] = 0.;
            for (int b = threadIdx.x; b < G; b += 32 * ns)
#pragma unroll
                for (int q = 0; q < K; ++q) t[q] += __ldcg(part + (size_t)q * G + b);
            warp_sums(t, st);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < K; ++q) {
            double t = st[0][q];
            for (int u = 1; u < ns; ++u) t += st[u][q];
            out[q] = dead ? __longlong_as_double(0x7ff8000000000000ll) : t;
        }
        // sm and st are written next after a barrier that follows these reads: sm is read only
        // before the second barrier above, st before the first barrier of the next reduction
    }

    // barrier only
    __device__ __forceinline__ void sync() {
        ++n;
        __syncthreads();
        int lost = 0;
        if (threadIdx.x == 0) lost = arrive_and_wait();
        if (__syncthreads_or(lost)) dead = true;
    }

  private:
    // counts this block in and polls until every block has: 1 when the wait ran out
    __device__ __forceinline__ int arrive_and_wait() {
        unsigned* ctr = reinterpret_cast<unsigned*>(slots);
        unsigned have;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
        int polls = dead ? GR_POLLS - 1 : 0;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(have) : "l"(ctr) : "memory");
        } while (have - n * (unsigned)gridDim.x > 0x7fffffffu && ++polls < GR_POLLS);
        return polls >= GR_POLLS;
    }
};

// The same sums with several blocks per SM and all partials added in block order (the three-sided
// momentum solve): block partials, barrier, totals.
constexpr int GR_ORDERED = 8;   // values of one such reduction at most
// doubles for a grid of `blocks` blocks: the counter's line, two buffers of partials after it
inline size_t gr_ordered_doubles(int blocks) { return 16 + (size_t)2 * GR_ORDERED * blocks; }
__device__ __forceinline__ double ldcg(const double* p) { return *p; }   // coherent load after a grid barrier

template <int K>
__device__ __forceinline__ void gr_warp_sum(double (&v)[K]) {
#pragma unroll
    for (int q = 0; q < K; ++q)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], off);
}

// block sums of v[0..K) into partials[blockIdx.x*GR_ORDERED + q]
template <int K>
__device__ void gr_block_partials(double (&v)[K], double* partials) {
    __shared__ double sm[GR_ORDERED][32];
    gr_warp_sum(v);
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < K; ++q) sm[q][w] = v[q];
    __syncthreads();
    if (w == 0) {
        double t[K];
#pragma unroll
        for (int q = 0; q < K; ++q) t[q] = lane < nw ? sm[q][lane] : 0.;
        gr_warp_sum(t);
        if (lane == 0)
#pragma unroll
            for (int q = 0; q < K; ++q) partials[blockIdx.x * GR_ORDERED + q] = t[q];
    }
    __syncthreads();
}

// sum of all blocks' partials, computed identically in every block; NaN after a lost wait
template <int K>
__device__ void gr_ordered_totals(const double* partials, bool lost, double (&out)[K]) {
    __shared__ double sm[GR_ORDERED][32];
    double v[K];
#pragma unroll
    for (int q = 0; q < K; ++q) v[q] = 0.;
    for (int g = threadIdx.x; g < (int)gridDim.x; g += blockDim.x)
#pragma unroll
        for (int q = 0; q < K; ++q) v[q] += ldcg(partials + (long long)g * GR_ORDERED + q);
    gr_warp_sum(v);
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < K; ++q) sm[q][w] = v[q];
    __syncthreads();
    if (w == 0) {
        double t[K];
#pragma unroll
        for (int q = 0; q < K; ++q) t[q] = lane < nw ? sm[q][lane] : 0.;
        gr_warp_sum(t);
        __syncwarp();
        if (lane == 0)
#pragma unroll
            for (int q = 0; q < K; ++q) sm[q][0] = lost ? __longlong_as_double(0x7ff8000000000000ll) : t[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < K; ++q) out[q] = sm[q][0];
    __syncthreads();
}

// Block partials, grid barrier, totals.  Partials alternate between two buffers: a block
// that races ahead to the next reduction cannot overwrite a slot another block is still
// summing, because it must first pass the barrier of the reduction in between.
template <int K>
__device__ __forceinline__ void gr_ordered_sum(GridRed& grid, double (&v)[K], double* partials, int& parity, double (&out)[K]) {
    double* buf = partials + (long long)(parity & 1) * gridDim.x * GR_ORDERED;
    gr_block_partials<K>(v, buf);
    grid.sync();
    gr_ordered_totals<K>(buf, grid.dead, out);
    ++parity;
}

}  // namespace cb
