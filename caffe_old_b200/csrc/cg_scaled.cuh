// Conjugate gradients on the symmetrically scaled 7-point operator: two streaming phases and one
// grid reduction per iteration.
//
// Jacobi-preconditioned CG on A (diagonal d of one sign, sigma) is plain CG on
//   B = sigma S A S,  S = |d|^(-1/2),  B y = sigma S b,  x = S y,
// whose diagonal is 1: a product reads three off-diagonal planes instead of four planes of A and
// one of 1/d.  The iterates are those of the preconditioned method; r of the text below is
// sigma S (b - A x), and (b - A x)^2 = |d| r^2 is summed beside (r, r) for the stopping test.
//
// The two reductions of an iteration merge (Meurant 1987):
//   update:   r -= alpha q;  p = r + beta p;  y += alpha p_old     (cell by cell)
//   barrier
//   product:  q = B p;  the sums (r, r), (p, q), (q, q)
// give alpha' = (r, r) / (p, q) and, as |r - alpha' q|^2 = alpha'^2 (q, q) - (r, r), the next beta
// before that residual exists.  The next update sums the residual itself, so the prediction
// never accumulates.  p is stored before the product, which then reads one vector at the stencil
// neighbours.
//
// Bytes per row and iteration (FP64): the update 64 (r, p, y read and written, q and d read), the
// product 40 (p, three planes, q): 104, on eight planes and no second buffers, so that half of a
// 2.1M-cell system stays in L2 between the phases (all of it in FP32); each phase sweeps from
// the end that the phase before it left there.  A thread takes W neighbouring cells, 16 bytes
// per load.
#pragma once
#include "gridred.cuh"

namespace cb {

// A projected solve of a singular system restarts when (r, r) has grown by this factor from its smallest:
// the round-off component of r along the null space never shrinks, and once the rest of r is down
// to it alpha and beta drive r up without end; the restart projects it away.  On singular
// 7-point systems (unit and lognormal conductances up to sigma 4, aspect ratios to 300) (r, r) rises by up
// to 7e4 in a sound solve.  Other systems don't restart on growth: with a nearly singular matrix
// (smallest eigenvalue 1e-9 of the diagonal) (r, r) rises further than this and then converges in 180 to 500
// iterations, which restarting turned into 4000 without convergence.
constexpr double CG_GROWTH = 1e6;

template <class T, int W> struct VecOf;
template <> struct VecOf<double, 1> { using type = double; };
template <> struct VecOf<double, 2> { using type = double2; };
template <> struct VecOf<float, 1> { using type = float; };
template <> struct VecOf<float, 4> { using type = float4; };

template <class T, int W>
__device__ __forceinline__ void ldw(const T* p, T (&v)[W]) {
    *reinterpret_cast<typename VecOf<T, W>::type*>(v) = *reinterpret_cast<const typename VecOf<T, W>::type*>(p);
}
template <class T, int W>
__device__ __forceinline__ void stw(T* p, const T (&v)[W]) {
    *reinterpret_cast<typename VecOf<T, W>::type*>(p) = *reinterpret_cast<const typename VecOf<T, W>::type*>(v);
}

// the same for data that is used once per iteration: first to leave L2
template <class T, int W>
__device__ __forceinline__ void ldw_once(const T* p, T (&v)[W]) {
    *reinterpret_cast<typename VecOf<T, W>::type*>(v) = __ldcs(reinterpret_cast<const typename VecOf<T, W>::type*>(p));
}
template <class T, int W>
__device__ __forceinline__ void stw_once(T* p, const T (&v)[W]) {
    __stcs(reinterpret_cast<typename VecOf<T, W>::type*>(p), *reinterpret_cast<const typename VecOf<T, W>::type*>(v));
}

template <class T>
struct CgVecs {
    T *r, *q, *p, *y;
    const T *E, *N, *U;   // off-diagonal planes of B: east, north, top
    const T* d;           // diagonal of A
    int n, nI, nIJ;
};

// Visits the groups of W cells of this thread, from the other end if `back`.  (Two groups at a time,
// for more loads in flight, spilled and was slower at every block size.)
template <int W, class F>
__device__ __forceinline__ void cg_groups(int n, bool back, F&& f) {
    const int groups = n / W, step = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
    const int steps = (groups + step - 1) / step;
    for (int s = 0; s < steps; ++s) {
        const int g = (back ? steps - 1 - s : s) * step + t0;
        if (g < groups) f(g * W);
    }
}

// r -= alpha q;  p = r + beta p;  y += alpha p_old;  sums (r, r) and (|d| r, r)
template <class T, int W>
__device__ __forceinline__ void cg_update(const CgVecs<T>& v, T alpha, T beta, bool back, double& rr, double& drr) {
    cg_groups<W>(v.n, back, [&](int c) {
        T R[W], Q[W], P[W], Y[W], D[W];
        ldw<T, W>(v.r + c, R); ldw<T, W>(v.q + c, Q); ldw<T, W>(v.p + c, P); ldw_once<T, W>(v.y + c, Y); ldw_once<T, W>(v.d + c, D);
#pragma unroll
        for (int m = 0; m < W; ++m) {
            R[m] = R[m] - alpha * Q[m];
            Y[m] = Y[m] + alpha * P[m];
            P[m] = R[m] + beta * P[m];
            const double s = (double)R[m] * R[m];
            rr += s;
            drr += fabs((double)D[m]) * s;
        }
        stw<T, W>(v.r + c, R); stw<T, W>(v.p + c, P); stw_once<T, W>(v.y + c, Y);
    });
}

// q = B p;  sums (p, q) and (q, q).  W > 1 needs nI and nI * nJ to be multiples of W, so that the
// neighbouring groups of a group are aligned.
template <class T, int W>
__device__ __forceinline__ void cg_product(const CgVecs<T>& v, bool back, double& pq, double& qq) {
    const T* p = v.p;
    cg_groups<W>(v.n, back, [&](int c) {
        T P[W], pN[W], pS[W], pT[W], pB[W], kE[W], kN[W], kS[W], kT[W], kB[W], Q[W];
        ldw<T, W>(p + c, P);
        ldw<T, W>(p + c + v.nI, pN); ldw<T, W>(p + c - v.nI, pS);
        ldw<T, W>(p + c + v.nIJ, pT); ldw<T, W>(p + c - v.nIJ, pB);
        const T w = p[c - 1], e = p[c + W], kw = v.E[c - 1];
        ldw<T, W>(v.E + c, kE);
        ldw<T, W>(v.N + c, kN); ldw<T, W>(v.N + c - v.nI, kS);
        ldw<T, W>(v.U + c, kT); ldw<T, W>(v.U + c - v.nIJ, kB);
#pragma unroll
        for (int m = 0; m < W; ++m) {
            Q[m] = P[m] + kE[m] * (m + 1 < W ? P[m + 1 < W ? m + 1 : 0] : e) + (m ? kE[m ? m - 1 : 0] : kw) * (m ? P[m ? m - 1 : 0] : w);
            Q[m] += kN[m] * pN[m] + kS[m] * pS[m];
            Q[m] += kT[m] * pT[m] + kB[m] * pB[m];
            pq += (double)P[m] * Q[m];
            qq += (double)Q[m] * Q[m];
        }
        stw<T, W>(v.q + c, Q);
    });
}

// alpha of the next update and the predicted beta, from t = (r, r), (p, q), (q, q); false on a
// breakdown
__device__ __forceinline__ bool cg_scalars(double rr, double pq, double qq, double& alpha, double& beta) {
    alpha = rr / pq;
    const double next = alpha * alpha * qq - rr;
    beta = next > 0. ? next / rr : 0.;
    return rr != 0. && pq != 0. && alpha == alpha && beta == beta;
}

}  // namespace cb
