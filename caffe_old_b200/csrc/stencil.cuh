// Stencil operators shared by the Krylov kernels: y = A x for the 7-point (momentum), the
// symmetric 7-point (pressure correction) and the compressed-row operators, with the
// immersed-boundary ghost rows, and the diagonal each preconditioner inverts.
#pragma once
#include "krylov.cuh"

namespace cb {

// Position in the ghost list of cell c, whose word is w (a search of the sorted list was a chain of
// about ten dependent loads, the longest path of a sweep over a lattice that one wave of threads covers).
__device__ __forceinline__ bool is_ghost(const uint2& w, long long c) { return (w.x >> (c & 31)) & 1u; }
__device__ __forceinline__ int ghost_index(const uint2& w, long long c) { return (int)w.y + __popc(w.x & ((1u << (c & 31)) - 1u)); }

// the row's 9 entries are loaded together, then the values they multiply
template <int NR, class X>
__device__ __forceinline__ void ghost_row(const GhostRows& gh, int g, X&& x, double (&y)[NR]) {
    int col[9];
    double val[9];
#pragma unroll
    for (int m = 0; m < 9; ++m) { col[m] = __ldg(gh.col + 9 * g + m); val[m] = __ldg(gh.val + 9 * g + m); }
#pragma unroll
    for (int q = 0; q < NR; ++q) {
        double s = 0.;
#pragma unroll
        for (int m = 0; m < 9; ++m)
            if (col[m] >= 0) s += val[m] * x(q, (long long)col[m]);
        y[q] = s;
    }
}
template <int NR, class X>
__device__ __forceinline__ void ghost_fix(const GhostRows& gh, const uint2& w, long long c, X&& x, double (&y)[NR]) {
    if (is_ghost(w, c)) ghost_row<NR>(gh, ghost_index(w, c), x, y);
}

template <int NR, class X>
__device__ __forceinline__ void apply(const Op7& A, long long c, X&& x, double (&y)[NR]) {
    const uint2 w = A.gh.n > 0 ? __ldg(A.gh.words + (c >> 5)) : make_uint2(0u, 0u);
    double aP = __ldg(A.a[0] + c), aE = __ldg(A.a[1] + c), aW = __ldg(A.a[2] + c), aN = __ldg(A.a[3] + c);
    double aS = __ldg(A.a[4] + c), aT = __ldg(A.a[5] + c), aB = __ldg(A.a[6] + c);
#pragma unroll
    for (int q = 0; q < NR; ++q)
        y[q] = aP * x(q, c) + aE * x(q, c + 1) + aW * x(q, c - 1) + aN * x(q, c + A.nI) + aS * x(q, c - A.nI)
               + aT * x(q, c + A.nIJ) + aB * x(q, c - A.nIJ);
    ghost_fix<NR>(A.gh, w, c, x, y);
}

template <int NR, class X>
__device__ __forceinline__ void apply(const OpSym& A, long long c, X&& x, double (&y)[NR]) {
    const uint2 w = A.gh.n > 0 ? __ldg(A.gh.words + (c >> 5)) : make_uint2(0u, 0u);
    double aP = __ldg(A.aP + c), aE = __ldg(A.aE + c), aW = __ldg(A.aE + c - 1), aN = __ldg(A.aN + c);
    double aS = __ldg(A.aN + c - A.nI), aT = __ldg(A.aT + c), aB = __ldg(A.aT + c - A.nIJ);
#pragma unroll
    for (int q = 0; q < NR; ++q)
        y[q] = aP * x(q, c) + aE * x(q, c + 1) + aW * x(q, c - 1) + aN * x(q, c + A.nI) + aS * x(q, c - A.nI)
               + aT * x(q, c + A.nIJ) + aB * x(q, c - A.nIJ);
    ghost_fix<NR>(A.gh, w, c, x, y);
}

template <int NR, class X>
__device__ __forceinline__ void apply(const OpCSR& A, long long c, X&& x, double (&y)[NR]) {
    const int p0 = __ldg(A.ptr + c), p1 = __ldg(A.ptr + c + 1);
#pragma unroll
    for (int q = 0; q < NR; ++q) y[q] = 0.;
    for (int p = p0; p < p1; ++p) {
        const double v = __ldg(A.val + p);
        const long long e = __ldg(A.col + p);
#pragma unroll
        for (int q = 0; q < NR; ++q) y[q] += v * x(q, e);
    }
}

__host__ __device__ __forceinline__ const double* diag_plane(const Op7& A) { return A.a[0]; }
__host__ __device__ __forceinline__ const double* diag_plane(const OpSym& A) { return A.aP; }
__device__ __forceinline__ double diag_of(const Op7& A, long long c) { return A.a[0][c]; }
__device__ __forceinline__ double diag_of(const OpCSR& A, long long c) {
    const int d = A.diag[c];
    return d >= 0 ? A.val[d] : 0.;
}
__device__ __forceinline__ double diag_of(const OpSym& A, long long c) { return A.aP[c]; }

}  // namespace cb
