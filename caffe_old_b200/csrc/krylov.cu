// Krylov solvers as persistent cooperative kernels.
//
// The reference calls PETSc (KSPBCGS + PCSOR, src/Math/SparseMatrix.cpp:86-106) once
// per system, from a zero initial guess, and returns the iteration count.  PETSc's
// lexicographic SOR sweep is sequential, so the device solvers use Jacobi
// preconditioning (the plain FP64 device path) with the published algorithms:
//   * BiCGStab (van der Vorst 1992), right-preconditioned, for the momentum system
//     (three right-hand sides sharing one operator sweep) and for non-symmetric
//     pressure-correction systems (immersed-boundary ghost rows);
//   * CG (Hestenes-Stiefel 1952) with one reduction per iteration (Meurant 1987) on the
//     symmetrically scaled system, for the symmetric pressure-correction system, and its
//     Chronopoulos-Gear form where that scaling does not apply.
// Every solve is one kernel launch: all blocks stay resident (cooperative launch) and
// meet in grid reductions between the phases of an iteration (gridred.cuh); every block
// sums the block partials in the same fixed order, so all blocks take the same
// convergence decision and the result is bit-reproducible.  The loop ends on the true
// residual ||b - A x|| <= rtol ||b|| (checked when the recursive residual meets it; the
// iteration restarts from the true residual otherwise) or at maxit, so no launch can run
// unbounded.  Lattices of at most 32768 cells, and compressed rows as far as they are short and few, run
// inside one cluster (krylov_small.cu).
//
// Values written earlier in the same launch by other blocks are read with ordinary loads
// after a reduction or barrier (whose release/acquire pair orders them), never through the
// read-only (non-coherent) path; only never-written inputs use __ldg.
#include <algorithm>
#include <cstring>
#include "bicgstab.cuh"
#include "cg_scaled.cuh"
#include "gridred.cuh"
#include "krylov.cuh"
#include "perdevice.h"
#include "stencil.cuh"

#define CAFFE_KSP_CG_JACOBI_INT 2   // caffe_ksp value of Jacobi-CG (include/caffe_b200.h)

namespace cb {

template <class Op>
__global__ void inv_diag_kernel(Op A, long long N, double* invD, double* slots) {
    gr_clear(slots);
    long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (c >= N) return;
    double dg = diag_of(A, c);
    invD[c] = dg != 0. ? 1. / dg : 1.;
}

template <class Op>
__device__ __forceinline__ void sym_row(const Op& A, long long c, double& aE, double& aN, double& aT, bool& ok);
template <>
__device__ __forceinline__ void sym_row(const OpSym& A, long long c, double& aE, double& aN, double& aT, bool& ok) {
    aE = A.aE[c]; aN = A.aN[c]; aT = A.aT[c];
}
template <>
__device__ __forceinline__ void sym_row(const Op7& A, long long c, double& aE, double& aN, double& aT, bool& ok) {
    aE = A.a[1][c]; aN = A.a[3][c]; aT = A.a[5][c];
}
// the west / south / bottom entries of row c equal the east / north / top ones of its neighbours
// (an entry whose neighbour lies outside the lattice is zero)
__device__ __forceinline__ bool row_symmetric(const OpSym&, long long, long long) { return true; }
__device__ __forceinline__ bool row_symmetric(const Op7& A, long long c, long long) {
    const double w = c >= 1 ? A.a[1][c - 1] : 0., s = c >= A.nI ? A.a[3][c - A.nI] : 0., b = c >= A.nIJ ? A.a[5][c - A.nIJ] : 0.;
    return A.a[2][c] == w && A.a[4][c] == s && A.a[6][c] == b;
}

// Planes of B = sigma S A S (cg_scaled.cuh): S and the east, north and top off-diagonals.  general
// (zero on entry) is set when the scaled form does not apply.
template <class Op, class T>
__global__ void scale_kernel(Op A, long long N, double* S, T* E, T* Nn, T* U, int* general, double* slots) {
    gr_clear(slots);
    long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (c >= N) return;
    const double d0 = diag_of(A, 0), d = diag_of(A, c);
    bool ok = (d0 > 0. && d > 0.) || (d0 < 0. && d < 0.);
    double aE, aN, aT;
    sym_row(A, c, aE, aN, aT, ok);
    ok = ok && row_symmetric(A, c, N);
    const double sg = d0 > 0. ? 1. : -1., s = 1. / sqrt(fabs(d));
    auto off = [&](double a, long long e) {   // a = 0 beyond the lattice's end
        return a == 0. ? 0. : e < N ? sg * a * s / sqrt(fabs(diag_of(A, e))) : __longlong_as_double(0x7ff8000000000000ll);
    };
    const double bE = off(aE, c + 1), bN = off(aN, c + A.nI), bT = off(aT, c + A.nIJ);
    ok = ok && s == s && bE == bE && bN == bN && bT == bT;
    S[c] = s; E[c] = (T)bE; Nn[c] = (T)bN; U[c] = (T)bT;
    if (!ok) *general = 1;
}

struct KArgs {
    const double* b;
    double* x;
    double* r;
    double* s;     // BiCGStab
    double* rp;
    double* p[2];
    double* v[2];
    double* t;
    const double* invD;
    double* partials;
    KspOut* out;
    long long N, PS;
    double rtol;
    double atol;   // absolute floor: converged when ||b - A x|| <= max(rtol ||b||, atol)
    int maxit;
    int project;   // remove the mean of b first (singular all-Neumann pressure systems)
    // fallback mode: when skip_if_ok is set the launch returns at once unless the status
    // it points to (the previous solve's) is non-zero; fallbacks counts the launches that ran
    const int* skip_if_ok;
    int* fallbacks;
    // CG: the scaled form's planes (1 / sqrt|d| in invD); null where only the general form runs
    double* cs[3];
};

// Whether the scaled CG may run, decided on the device by scale_kernel: every diagonal entry of
// one sign and, for seven separate coefficient planes, a symmetric matrix.
__device__ __forceinline__ bool scaled_form(const KspOut* o) { return o->general == 0; }

// Remove the mean of b (one plane), in place; every block computes the same mean.  Twice: where b was
// almost a constant, what the first pass leaves is as much the rounding of that mean as b, and a
// component along the null space that no iteration can remove makes CG diverge once r is down to it.
__device__ __forceinline__ void project_mean(GridRed& grid, double* b, long long N, long long t0, long long T) {
    for (int pass = 0; pass < 2; ++pass) {
        double s[1] = {0.};
        for (long long c = t0; c < N; c += T) s[0] += b[c];
        double tot[1];
        grid.sum<1>(s, tot);
        double mean = tot[0] / (double)N;
        for (long long c = t0; c < N; c += T) b[c] = b[c] - mean;
    }
    // the projected b is read at stencil neighbours owned by other blocks right after this
    // (CG forms w = A D^-1 b): every block's subtraction must be visible first
    grid.sync();
}

// ------------------------------------------------------------------ BiCGStab
// Right-preconditioned BiCGStab (van der Vorst 1992) with two sweeps and two grid reductions per
// iteration.  The vectors are stored as D^-1 times themselves (R, S, T, P, V for r, s, t, p, v), the form in
// which the operator takes them, so that no 1/d is read at the stencil neighbours:
//   sweep 1:  x += alpha P + omega S;  R = S - omega T;  P' = R + beta (P - omega V);  v = A P';  (rp, v)
//   sweep 2:  S = R - alpha V;  t = A S;  (t, s), (t, t), (rp, s), (rp, t), (s, s)
// The last sums give omega and, as r = s - omega t, the next rho = (rp, s) - omega (rp, t) and
// (r, r) = (s, s) - 2 omega (t, s) + omega^2 (t, t) without a third sweep and reduction.  P' and S
// are formed at the stencil neighbours from the stored vectors; P and V are double-buffered.
// At a check (the recursive norm meets the tolerance, maxit, a breakdown) x takes the half-finished
// iteration's update and the true residual decides, as in CG.
// y = A x of one row for the two sweeps.  What bounds a sweep at 40^3 to 100^3 is the chain of loads of
// each step (2.5 us a step): a row's own values are loaded ahead of the product and the product's
// operands before its first operation.  One cell per thread: pairs of cells halve the steps, but leave
// half the loads in flight at the same registers and run the two cells' ghost rows one after the
// other (us per iteration, FP64, sphere: 64x44x42 10.0 against 12.3, 80x52x50 12.9 against 14.7,
// 96x64x64 16.8 against 21.1; 13.0 against 13.2 at 72x48x48 and, with the loads in the order of use, 10.3
// against 13.5 at 75x39x41).  Ghost rows stay in the sweep: as items of their own after the stencil
// rows they took 13.6 at 75x39x41 and 21.2 at 96x64x64.
template <class Op, class X>
__device__ __forceinline__ double row_product(const Op& A, long long c, X&& x) { double y[1]; apply<1>(A, c, x, y); return y[0]; }
// every operand asked for before the first one is used
template <class X>
__device__ __forceinline__ double row_product(const OpSym& A, long long c, X&& x) {
    const uint2 g = A.gh.n > 0 ? __ldg(A.gh.words + (c >> 5)) : make_uint2(0u, 0u);
    const double o = x(0, c), n = x(0, c + A.nI), s = x(0, c - A.nI), t = x(0, c + A.nIJ), b = x(0, c - A.nIJ);
    const double w = x(0, c - 1), e = x(0, c + 1), kW = A.aE[c - 1];
    const double kP = A.aP[c], kE = A.aE[c], kN = A.aN[c], kS = A.aN[c - A.nI], kT = A.aT[c], kB = A.aT[c - A.nIJ];
    double y = kP * o + kE * e + kW * w + kN * n + kS * s + kT * t + kB * b;
    if (is_ghost(g, c)) { double v[1]; ghost_row<1>(A.gh, ghost_index(g, c), x, v); y = v[0]; }
    return y;
}

struct BiVecs {
    double *x, *r, *s, *t, *rp;
    const double* invD;
    long long N, t0, T;   // rows, this thread's first, and the step
};

// sweep 1:  x += xa P + xo S;  R = S - omega T;  P' = R + beta (P - omega V);  v = A P';  sum (rp, v)
template <class Op>
__device__ __forceinline__ double bi_sweep1(const Op& A, const BiVecs& b, const double* P, const double* V, double* Pn, double* Vn,
                                            double alpha, double omega, double beta) {
    double acc = 0.;
    auto next = [&](int, long long e) { return (b.s[e] - omega * b.t[e]) + beta * (P[e] - omega * V[e]); };
    for (long long c = b.t0; c < b.N; c += b.T) {
        const double id = b.invD[c], x = b.x[c], rp = b.rp[c];
        const double y = row_product(A, c, next);
        const double s = b.s[c], t = b.t[c], p = P[c], v = V[c];
        const double r = s - omega * t;
        b.x[c] = x + (alpha * p + omega * s);
        b.r[c] = r;
        Pn[c] = r + beta * (p - omega * v);
        Vn[c] = id * y;
        acc += rp * y;
    }
    return acc;
}

// sweep 2:  S = R - alpha V;  t = A S;  sums (t, s), (t, t), (rp, s), (rp, t), (s, s)
template <class Op>
__device__ __forceinline__ void bi_sweep2(const Op& A, const BiVecs& b, const double* V, double alpha, double (&acc)[5]) {
    auto next = [&](int, long long e) { return b.r[e] - alpha * V[e]; };
    for (long long c = b.t0; c < b.N; c += b.T) {
        const double id = b.invD[c], d = diag_of(A, c), rp = b.rp[c];
        const double t = row_product(A, c, next);
        const double S = b.r[c] - alpha * V[c], s = (d != 0. ? d : 1.) * S;
        b.s[c] = S;
        b.t[c] = id * t;
        acc[0] += t * s; acc[1] += t * t; acc[2] += rp * s; acc[3] += rp * t; acc[4] += s * s;
    }
}

// omega, next beta and rho, and (r, r) from the sums of sweep 2; true when the iteration may go on with
// them (bi_sound)
__device__ __forceinline__ bool bi_scalars(const double* t, double rp2, double alpha, double& omega, double& beta, double& rho, double& rr) {
    omega = t[1] == 0. ? 0. : t[0] / t[1];
    const double rn = t[2] - omega * t[3];
    rr = t[4] - 2. * omega * t[0] + omega * omega * t[1];
    beta = (rn / rho) * (alpha / omega);
    rho = rn;
    return omega != 0. && rr == rr && bi_sound(rn, rp2, rr);
}

template <class Op>
__global__ void __launch_bounds__(512) bicgstab_kernel(Op A, KArgs a) {
    if (a.skip_if_ok && *a.skip_if_ok == 0) return;   // uniform across the grid: no barrier is reached
    if (a.skip_if_ok && blockIdx.x == 0 && threadIdx.x == 0 && a.fallbacks) atomicAdd(a.fallbacks, 1);
    GridRed grid(a.partials);
    const long long N = a.N;
    const long long T = (long long)gridDim.x * blockDim.x;
    const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const double* invD = a.invD;
    if (a.project) project_mean(grid, const_cast<double*>(a.b), N, t0, T);
    // ---- initial state: x = 0, r = rp = b (S holds it for the first sweep, with P = V = T = 0)
    double bb[1];
    {
        double acc[1] = {0.};
        for (long long c = t0; c < N; c += T) {
            const double bv = a.b[c];
            a.x[c] = 0.;
            a.s[c] = invD[c] * bv;
            a.rp[c] = bv;
            a.t[c] = 0.; a.p[0][c] = 0.; a.v[0][c] = 0.;
            acc[0] += bv * bv;
        }
        grid.sum<1>(acc, bb);
    }
    double rho = bb[0], rp2 = bb[0], alpha = 0., omega = 0., beta = 0., relres = 0.;
    const double tol2 = fmax(a.rtol * a.rtol * bb[0], a.atol * a.atol);
    int it = 0, status = bb[0] != bb[0] ? 3 : 0;
    // x = 0 already meets the absolute floor: nothing to do (relative residual 1)
    bool done = !(bb[0] > 0.) || bb[0] <= tol2;
    if (bb[0] > 0. && done) relres = 1.;
    BiVecs v;
    v.x = a.x; v.r = a.r; v.s = a.s; v.t = a.t; v.rp = a.rp; v.invD = invD; v.N = N;
    v.t0 = t0; v.T = T;
    int cur = 0;
    while (!done) {
        double rv[1], acc1[1];
        acc1[0] = bi_sweep1(A, v, a.p[cur], a.v[cur], a.p[cur ^ 1], a.v[cur ^ 1], alpha, omega, beta);
        grid.sum<1>(acc1, rv);
        alpha = omega = 0.;   // x is up to date with R
        cur ^= 1;
        const bool broke = rv[0] == 0. || rv[0] != rv[0];
        if (!broke) {
            alpha = rho / rv[0];
            double acc[5] = {0., 0., 0., 0., 0.}, tot[5], rr;
            bi_sweep2(A, v, a.v[cur], alpha, acc);
            grid.sum<5>(acc, tot);
            it += 1;
            const bool sound = bi_scalars(tot, rp2, alpha, omega, beta, rho, rr);
            if (sound && rr > tol2 && it < a.maxit) continue;
            for (long long c = t0; c < N; c += T) a.x[c] = a.x[c] + (alpha * a.p[cur][c] + omega * a.s[c]);
            grid.sync();
        } else
            it += 1;   // a breakdown counts: from the same residual it repeats, and maxit must end it
        // ---- true residual r = b - A x.  After a breakdown x is what it was: P' may not be finite there
        double acc[1] = {0.}, rrT[1];
        for (long long c = t0; c < N; c += T) {
            double y[1];
            apply<1>(A, c, [&](int, long long e) { return a.x[e]; }, y);
            const double rt = a.b[c] - y[0];
            a.s[c] = invD[c] * rt; a.rp[c] = rt;
            a.t[c] = 0.; a.p[cur][c] = 0.; a.v[cur][c] = 0.;
            acc[0] += rt * rt;
        }
        grid.sum<1>(acc, rrT);
        relres = sqrt(rrT[0] / bb[0]);
        if (rrT[0] <= tol2) { done = true; status = 0; }
        else if (rrT[0] != rrT[0]) { done = true; status = 3; }
        else if (it >= a.maxit) { done = true; status = 1; }
        else { rho = rp2 = rrT[0]; alpha = omega = beta = 0.; }   // restart from the true residual
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) { a.out->iters[0] = it; a.out->relres[0] = relres; a.out->status[0] = status; }
}

// ------------------------------------------------------------------ BiCGStab, three right-hand sides
// The momentum solve: three right-hand sides share one operator sweep.  Classic order of the method,
// three sweeps and reductions per iteration: with three right-hand sides the two-sweep form needs 15
// sums and twelve vectors at the stencil neighbours, spills at 128 registers and takes the same time
// (0.36 against 0.38 ms per iteration at 128^3), and a solve is 3 to 15 iterations.  Two blocks of KB
// threads per SM, partials summed in block order.
constexpr int KB = 256;   // threads per block
constexpr int KB_PER_SM = 2;

template <int NR, class Op>
__global__ void __launch_bounds__(KB, KB_PER_SM) bicgstab3_kernel(Op A, KArgs a) {
    GridRed grid(a.partials);
    const long long N = a.N, PS = a.PS;
    const long long T = (long long)gridDim.x * blockDim.x;
    const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const double* invD = a.invD;

    double acc[2 * NR];
    int par = 0;
    // ---- initial state: x = 0, r = rp = b
#pragma unroll
    for (int q = 0; q < NR; ++q) acc[q] = 0.;
    for (long long c = t0; c < N; c += T) {
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            double bv = a.b[q * PS + c];
            a.x[q * PS + c] = 0.;
            a.r[q * PS + c] = bv;
            a.rp[q * PS + c] = bv;
            acc[q] += bv * bv;
        }
    }
    double bb[NR];
    {
        double tmp[NR];
#pragma unroll
        for (int q = 0; q < NR; ++q) tmp[q] = acc[q];
        gr_ordered_sum<NR>(grid, tmp, a.partials + 16, par, bb);
    }

    double rho[NR], rho_old[NR], alpha[NR], omega[NR], tol2[NR];
    int it[NR], status[NR];
    bool done[NR], fresh[NR], needT[NR];
    double relres[NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) {
        rho[q] = bb[q]; rho_old[q] = 1.; alpha[q] = 1.; omega[q] = 1.;
        tol2[q] = fmax(a.rtol * a.rtol * bb[q], a.atol * a.atol);
        it[q] = 0; fresh[q] = true; needT[q] = false; relres[q] = 0.;
        // x = 0 already meets the absolute floor: nothing to do (relative residual 1)
        done[q] = !(bb[q] > 0.) || bb[q] <= tol2[q];
        if (bb[q] > 0. && done[q]) relres[q] = 1.;
        if (bb[q] != bb[q]) status[q] = 3; else status[q] = 0;
    }
    int cur = 0;
    while (true) {
        bool run[NR], any = false;
#pragma unroll
        for (int q = 0; q < NR; ++q) { run[q] = !done[q]; any |= run[q]; }
        if (!any) break;
        double beta[NR];
#pragma unroll
        for (int q = 0; q < NR; ++q) beta[q] = fresh[q] ? 0. : (rho[q] / rho_old[q]) * (alpha[q] / omega[q]);
        const double* po = a.p[cur];
        const double* vo = a.v[cur];
        double* pn = a.p[cur ^ 1];
        double* vn = a.v[cur ^ 1];
        // ---- phase 1: p = r + beta (p_old - omega v_old);  v = A D^-1 p;  (rp, v)
#pragma unroll
        for (int q = 0; q < NR; ++q) acc[q] = 0.;
        for (long long c = t0; c < N; c += T) {
            auto pnew = [&](int q, long long e) -> double {
                double rv = ldcg(a.r + q * PS + e);
                if (fresh[q]) return rv;
                return rv + beta[q] * (ldcg(po + q * PS + e) - omega[q] * ldcg(vo + q * PS + e));
            };
            double y[NR];
            apply<NR>(A, c, [&](int q, long long e) { return __ldg(invD + e) * pnew(q, e); }, y);
#pragma unroll
            for (int q = 0; q < NR; ++q) {
                if (!run[q]) continue;
                double pc = pnew(q, c);
                pn[q * PS + c] = pc;
                vn[q * PS + c] = y[q];
                double rpv;
                if (fresh[q]) { rpv = ldcg(a.r + q * PS + c); a.rp[q * PS + c] = rpv; }
                else rpv = a.rp[q * PS + c];
                acc[q] += rpv * y[q];
            }
        }
        double rv[NR];
        {
            double tmp[NR];
#pragma unroll
            for (int q = 0; q < NR; ++q) tmp[q] = acc[q];
            gr_ordered_sum<NR>(grid, tmp, a.partials + 16, par, rv);
        }
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            if (!run[q]) continue;
            if (rv[q] == 0. || rv[q] != rv[q]) { needT[q] = true; run[q] = false; it[q] += 1; }   // counted: a breakdown may repeat
            else alpha[q] = rho[q] / rv[q];
        }
        // ---- phase 2: s = r - alpha v;  t = A D^-1 s;  (t, s), (t, t)
#pragma unroll
        for (int q = 0; q < 2 * NR; ++q) acc[q] = 0.;
        for (long long c = t0; c < N; c += T) {
            double y[NR];
            apply<NR>(A, c, [&](int q, long long e) {
                return __ldg(invD + e) * (ldcg(a.r + q * PS + e) - alpha[q] * ldcg(vn + q * PS + e));
            }, y);
#pragma unroll
            for (int q = 0; q < NR; ++q) {
                if (!run[q]) continue;
                double s = ldcg(a.r + q * PS + c) - alpha[q] * ldcg(vn + q * PS + c);
                a.t[q * PS + c] = y[q];
                acc[2 * q] += y[q] * s;
                acc[2 * q + 1] += y[q] * y[q];
            }
        }
        double tot[2 * NR];
        {
            double tmp[2 * NR];
#pragma unroll
            for (int q = 0; q < 2 * NR; ++q) tmp[q] = acc[q];
            gr_ordered_sum<2 * NR>(grid, tmp, a.partials + 16, par, tot);
        }
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            if (!run[q]) continue;
            omega[q] = tot[2 * q + 1] == 0. ? 0. : tot[2 * q] / tot[2 * q + 1];
        }
        // ---- phase 3: x += alpha D^-1 p + omega D^-1 s;  r = s - omega t;  (r, rp), (r, r)
#pragma unroll
        for (int q = 0; q < 2 * NR; ++q) acc[q] = 0.;
        for (long long c = t0; c < N; c += T) {
            double id = __ldg(invD + c);
#pragma unroll
            for (int q = 0; q < NR; ++q) {
                if (!run[q]) continue;
                double s = ldcg(a.r + q * PS + c) - alpha[q] * ldcg(vn + q * PS + c);
                double ph = id * ldcg(pn + q * PS + c);
                double sh = id * s;
                a.x[q * PS + c] = a.x[q * PS + c] + (alpha[q] * ph + omega[q] * sh);
                double rn = s - omega[q] * ldcg(a.t + q * PS + c);
                a.r[q * PS + c] = rn;
                acc[2 * q] += rn * a.rp[q * PS + c];
                acc[2 * q + 1] += rn * rn;
            }
        }
        {
            double tmp[2 * NR];
#pragma unroll
            for (int q = 0; q < 2 * NR; ++q) tmp[q] = acc[q];
            gr_ordered_sum<2 * NR>(grid, tmp, a.partials + 16, par, tot);
        }
        bool anyT = false;
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            if (run[q]) {
                it[q] += 1;
                fresh[q] = false;
                rho_old[q] = rho[q];
                rho[q] = tot[2 * q];
                double rr = tot[2 * q + 1];
                if (rr <= tol2[q] || omega[q] == 0. || it[q] >= a.maxit || rr != rr) needT[q] = true;
            }
            anyT |= needT[q];
        }
        cur ^= 1;
        if (anyT) {
            // ---- true residual r = b - A x for the components being checked
#pragma unroll
            for (int q = 0; q < NR; ++q) acc[q] = 0.;
            for (long long c = t0; c < N; c += T) {
                double y[NR];
                apply<NR>(A, c, [&](int q, long long e) { return ldcg(a.x + q * PS + e); }, y);
#pragma unroll
                for (int q = 0; q < NR; ++q) {
                    if (!needT[q]) continue;
                    double rt = a.b[q * PS + c] - y[q];
                    a.r[q * PS + c] = rt;
                    acc[q] += rt * rt;
                }
            }
            double rrT[NR];
            {
                double tmp[NR];
#pragma unroll
                for (int q = 0; q < NR; ++q) tmp[q] = acc[q];
                gr_ordered_sum<NR>(grid, tmp, a.partials + 16, par, rrT);
            }
#pragma unroll
            for (int q = 0; q < NR; ++q) {
                if (!needT[q]) continue;
                needT[q] = false;
                relres[q] = sqrt(rrT[q] / bb[q]);
                if (rrT[q] <= tol2[q]) { done[q] = true; status[q] = 0; }
                else if (rrT[q] != rrT[q]) { done[q] = true; status[q] = 3; }
                else if (it[q] >= a.maxit) { done[q] = true; status[q] = 1; }
                else { fresh[q] = true; rho[q] = rrT[q]; rho_old[q] = 1.; alpha[q] = 1.; omega[q] = 1.; }
            }
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        for (int q = 0; q < NR; ++q) { a.out->iters[q] = it[q]; a.out->relres[q] = relres[q]; a.out->status[q] = status[q]; }
    }
}

// ------------------------------------------------------------------ CG, one reduction per iteration
// Chronopoulos & Gear (1989) form of preconditioned CG: with u = M^-1 r and w = A u the two
// inner products (r, u) and (w, u) are taken together, so an iteration is one sweep and one
// grid barrier:
//   s_i = w_i + beta_i s_{i-1};  p_i = u_i + beta_i p_{i-1};  x += alpha_i p_i;
//   r_{i+1} = r_i - alpha_i s_i;  u_{i+1} = M^-1 r_{i+1};  w_{i+1} = A u_{i+1};
//   gamma = (r_{i+1}, u_{i+1}), delta = (w_{i+1}, u_{i+1});
//   beta_{i+1} = gamma_{i+1} / gamma_i;  alpha_{i+1} = gamma_{i+1} / (delta - beta_{i+1} gamma_{i+1} / alpha_i).
// u_{i+1} at the stencil neighbours is recomputed from r_i, w_i and s_{i-1}, which are
// double-buffered (the sweep writes the other buffer).
template <class Op>
__global__ void __launch_bounds__(1024) cg1_kernel(Op A, KArgs a) {
    if (a.skip_if_ok && *a.skip_if_ok == 0) return;   // uniform across the grid: no barrier is reached
    if (a.cs[0] && scaled_form(a.out)) return;        // cgs_kernel ran
    if (a.skip_if_ok && blockIdx.x == 0 && threadIdx.x == 0 && a.fallbacks) atomicAdd(a.fallbacks, 1);
    GridRed grid(a.partials);
    const long long N = a.N, PS = a.PS;
    const long long T = (long long)gridDim.x * blockDim.x;
    const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const double* invD = a.invD;
    // current (read) and next (written) buffers, swapped after every sweep
    double *rC = a.r, *rN = a.r + PS, *wC = a.v[0], *wN = a.v[1], *sC = a.p[0], *sN = a.p[1];
    double* p = a.t;       // u = M^-1 r is not stored: it is recomputed from r where needed
    if (a.project) project_mean(grid, const_cast<double*>(a.b), N, t0, T);
    // ---- start: x = 0, r = b, u = M^-1 b, w = A u, s_-1 = p_-1 = 0
    double acc[3] = {0., 0., 0.};
    for (long long c = t0; c < N; c += T) {
        double bv = a.b[c];
        double uv = __ldg(invD + c) * bv;
        double y[1];
        apply<1>(A, c, [&](int, long long e) { return __ldg(invD + e) * a.b[e]; }, y);
        a.x[c] = 0.;
        rC[c] = bv; wC[c] = y[0]; sC[c] = 0.; p[c] = 0.;
        acc[0] += bv * uv; acc[1] += y[0] * uv; acc[2] += bv * bv;
    }
    double tot[3];
    grid.sum<3>(acc, tot);
    double gamma = tot[0], bb = tot[2];
    double tol2 = fmax(a.rtol * a.rtol * bb, a.atol * a.atol);
    double alpha = tot[1] != 0. ? gamma / tot[1] : 0., beta = 0.;
    int it = 0, status = 0;
    double relres = 0.;
    bool done = !(bb > 0.) || bb <= tol2;   // x = 0 already meets the absolute floor
    if (bb > 0. && done) relres = 1.;
    if (bb != bb) status = 3;
    while (!done) {
        const double* r0 = rC;
        const double* w0 = wC;
        const double* s0 = sC;
        double* r1 = rN;
        double* w1 = wN;
        double* s1 = sN;
        acc[0] = acc[1] = acc[2] = 0.;
        for (long long c = t0; c < N; c += T) {
            double idc = __ldg(invD + c);
            double r0c = r0[c];
            double si = w0[c] + beta * s0[c];
            double pi = idc * r0c + beta * p[c];
            a.x[c] = a.x[c] + alpha * pi;
            double rn = r0c - alpha * si;
            double un = idc * rn;
            double y[1];
            apply<1>(A, c, [&](int, long long e) {
                return __ldg(invD + e) * (r0[e] - alpha * (w0[e] + beta * s0[e]));
            }, y);
            s1[c] = si; p[c] = pi; r1[c] = rn; w1[c] = y[0];
            acc[0] += rn * un; acc[1] += y[0] * un; acc[2] += rn * rn;
        }
        grid.sum<3>(acc, tot);
        it += 1;
        { double* t_ = rC; rC = rN; rN = t_; t_ = wC; wC = wN; wN = t_; t_ = sC; sC = sN; sN = t_; }
        double gn = tot[0], dn = tot[1], rr = tot[2];
        bool check = rr <= tol2 || it >= a.maxit || rr != rr;
        double bn = gn / gamma;
        double den = dn - bn * gn / alpha;
        if (den == 0. || den != den || gamma == 0.) check = true;
        beta = bn; alpha = gn / den; gamma = gn;
        if (check) {
            // ---- true residual r = b - A x (into the current buffer)
            double* rc = rC;
            double a2[1] = {0.};
            for (long long c = t0; c < N; c += T) {
                double y[1];
                apply<1>(A, c, [&](int, long long e) { return a.x[e]; }, y);
                double rt = a.b[c] - y[0];
                rc[c] = rt;
                a2[0] += rt * rt;
            }
            double t1[1];
            grid.sum<1>(a2, t1);
            relres = sqrt(t1[0] / bb);
            if (t1[0] <= tol2) { done = true; status = 0; }
            else if (t1[0] != t1[0]) { done = true; status = 3; }
            else if (it >= a.maxit) { done = true; status = 1; }
            else {
                // restart from the true residual: u = M^-1 r, w = A u, s = p = 0
                double a3[2] = {0., 0.};
                double* wc = wC;
                double* sc = sC;
                for (long long c = t0; c < N; c += T) {
                    double uv = __ldg(invD + c) * rc[c];
                    double y[1];
                    apply<1>(A, c, [&](int, long long e) { return __ldg(invD + e) * rc[e]; }, y);
                    wc[c] = y[0]; sc[c] = 0.; p[c] = 0.;
                    a3[0] += rc[c] * uv; a3[1] += y[0] * uv;
                }
                double t2[2];
                grid.sum<2>(a3, t2);
                gamma = t2[0];
                alpha = t2[1] != 0. ? gamma / t2[1] : 0.;
                beta = 0.;
                if (gamma == 0.) { done = true; status = 2; }
            }
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) { a.out->iters[0] = it; a.out->relres[0] = relres; a.out->status[0] = status; }
}

// ------------------------------------------------------------------ CG, scaled form
// The solve's frame around cg_update and cg_product: start, true-residual check, restart and unscaling as in
// cg1_kernel, which runs instead where the scaled form does not apply.
template <class Op, int W>
__global__ void __launch_bounds__(1024) cgs_kernel(Op A, KArgs a) {
    if (a.skip_if_ok && *a.skip_if_ok == 0) return;
    if (!scaled_form(a.out)) return;
    if (a.skip_if_ok && blockIdx.x == 0 && threadIdx.x == 0 && a.fallbacks) atomicAdd(a.fallbacks, 1);
    GridRed grid(a.partials);
    const long long N = a.N;
    const long long T = (long long)gridDim.x * blockDim.x;
    const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const double* S = a.invD;
    const double sg = diag_of(A, 0) > 0. ? 1. : -1.;
    CgVecs<double> v;
    v.r = a.r; v.q = a.v[0]; v.p = a.p[0]; v.y = a.x;
    v.E = a.cs[0]; v.N = a.cs[1]; v.U = a.cs[2];
    v.d = diag_plane(A);
    v.n = (int)N; v.nI = (int)A.nI; v.nIJ = (int)A.nIJ;
    if (a.project) project_mean(grid, const_cast<double*>(a.b), N, t0, T);
    double bb;
    {
        double s[1] = {0.}, tot[1];
        for (long long c = t0; c < N; c += T) {
            const double bv = a.b[c];
            v.r[c] = sg * S[c] * bv; v.q[c] = 0.; v.p[c] = 0.; v.y[c] = 0.;
            s[0] += bv * bv;
        }
        grid.sum<1>(s, tot);
        bb = tot[0];
    }
    const double tol2 = fmax(a.rtol * a.rtol * bb, a.atol * a.atol);
    int it = 0, status = 0;
    double relres = 0.;
    bool done = !(bb > 0.) || bb <= tol2;   // x = 0 already meets the absolute floor
    if (bb > 0. && done) relres = 1.;
    if (bb != bb) status = 3;
    double alpha = 0., beta = 0., best = bb;
    bool first = true;                      // the first update forms p = r only
    while (!done) {
        double acc[4] = {0., 0., 0., 0.}, tot[4];
        cg_update<double, W>(v, alpha, beta, false, acc[0], acc[1]);
        grid.sync();
        cg_product<double, W>(v, true, acc[2], acc[3]);
        grid.sum<4>(acc, tot);
        if (!first) ++it;
        const bool broke = !cg_scalars(tot[0], tot[2], tot[3], alpha, beta);
        const bool stuck = broke && first;   // no direction from a fresh residual: a restart would not help
        if (tot[1] < best) best = tot[1];
        if ((!first && (tot[1] <= tol2 || it >= a.maxit)) || tot[1] != tot[1] || (a.project && tot[1] > CG_GROWTH * best) || broke) {
            // ---- true residual r = b - A x, x = S y
            double s[3] = {0., 0., 0.}, t[3];
            for (long long c = t0; c < N; c += T) {
                double y[1];
                apply<1>(A, c, [&](int, long long e) { return S[e] * v.y[e]; }, y);
                const double rt = a.b[c] - y[0], rs = sg * S[c] * rt;
                v.r[c] = rs; v.q[c] = 0.; v.p[c] = 0.;
                s[0] += rt * rt; s[1] += rs * rs; s[2] += rt;
            }
            grid.sum<3>(s, t);
            relres = sqrt(t[0] / bb);
            if (t[0] <= tol2) { done = true; status = 0; }
            else if (t[0] != t[0]) { done = true; status = 3; }
            else if (it >= a.maxit) { done = true; status = 1; }
            else if (stuck || t[1] == 0.) { done = true; status = 2; }
            alpha = beta = 0.;   // restart from the true residual, in the range of a singular A
            first = true;
            best = t[0];
            if (a.project)   // by the thread whose update reads the cell next
                cg_groups<W>(v.n, false, [&](int c) {
#pragma unroll
                    for (int m = 0; m < W; ++m) v.r[c + m] = v.r[c + m] - sg * S[c + m] * (t[2] / (double)N);
                });
        } else
            first = false;
    }
    for (long long c = t0; c < N; c += T) a.x[c] = S[c] * v.y[c];
    if (blockIdx.x == 0 && threadIdx.x == 0) { a.out->iters[0] = it; a.out->relres[0] = relres; a.out->status[0] = status; }
}

// ------------------------------------------------------------------ mixed precision
// FP32 CG inside FP64 iterative refinement (the precision form of the pressure correction): the
// true residual r = b - A x, the update x += e, and every dot product and norm stay FP64; the scaled
// operator's planes, the Krylov vectors and the operator sweeps are FP32.  One launch runs the whole
// solve.
//
// A refinement does not restart the Krylov process (Sleijpen & van der Vorst 1996, reliable
// updates): whenever the recursive residual has fallen by MX_DROP since the last one, x takes the
// FP32 correction, the FP64 residual replaces the recursive one, and the iteration goes on with the
// search direction it has.  Restarting instead cost the 128^3 skewed cavity 1950 iterations a
// step against 1680, as many as in FP64.  A recursive residual that has left the true one, or
// MX_PATIENCE iterations without a new smallest residual, count as a stall: the process restarts from
// the true residual, and the second stall in a row leaves the solve to the FP64 fallback.
//
// Symmetric systems only.  With immersed-boundary ghost rows the mixed form runs the FP64 BiCGStab: FP32
// BiCGStab loses its biorthogonality there.  Measured on 72x48x48 and 75x39x41 sphere cases (FP64
// 4719 and 5690 iterations a step, 66 and 76 ms): FP32 to 1e-6 and restarted, stalled in every
// solve, then the FP64 solve, 0.5-1.2 s; FP32 with reliable updates 24829 and 23281 iterations, 547
// and 266 ms; FP64 vectors on the FP32 matrix 12772 and 10529, 171 and 160 ms.
//
// Both figures measured on a skewed 128^3 cavity (3 steps, 5724 iterations) and on one of 64x60x56 cells in a
// box of 1 x 0.02 x 0.2 (4 steps, 91,740), ms of the p' solves.  MX_DROP 0.5: 100 and 484; 0.2: 96 and 506; 0.05: 94 and
// 591; 0.01: 94 and 736; 0.001: 101 and 590.  Patience 300 leaves four of the second cavity's eight solves
// to FP64 (1104 ms); 3000 changes neither (94 and 606) and takes longer to give up.
constexpr double MX_DROP = 0.05;
constexpr int MX_PATIENCE = 1000;

__global__ void cast_kernel(long long N, const double* d, float* f) {
    long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (c < N) f[c] = (float)d[c];
}

struct MxArgs {
    const double* b;
    double* x;
    float *r, *q, *p, *e;
    const float* d;         // the diagonal
    const float* cs[3];     // the scaled operator's planes
    const double* S;        // 1 / sqrt|d|
    double* partials;
    KspOut* out;
    long long N;
    double rtol;
    double atol;
    int maxit;
    int project;
};

// Watches the residual norms.
struct MxWatch {
    double tol2, best, top;      // ||r||^2: tolerance, smallest so far, largest since the last refinement
    int since = 0, stalls = 0;   // iterations since the smallest, stalls in a row
    __device__ void start(double rr) { best = top = rr; }
    // after an iteration: whether to refine now
    __device__ bool due(double rr) {
        if (rr < best) { best = rr; since = 0; stalls = 0; } else ++since;
        if (rr > top) top = rr;
        return rr <= tol2 || rr <= MX_DROP * MX_DROP * top || since >= MX_PATIENCE || rr != rr;
    }
    // at a refinement from the recursive rr to the true one: whether the process has to restart
    __device__ bool refine(double rr, double truth) {
        const bool stalled = since >= MX_PATIENCE || !(fabs(rr) > 0.25 * truth && fabs(rr) < 4. * truth);
        if (stalled) { ++stalls; since = 0; best = truth; }
        top = truth;
        return stalled;
    }
};

template <int W>
__global__ void __launch_bounds__(1024) mixed_cg_kernel(OpSym A, MxArgs a) {
    GridRed grid(a.partials);
    const long long N = a.N, T = (long long)gridDim.x * blockDim.x, t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const double sg = diag_of(A, 0) > 0. ? 1. : -1.;
    CgVecs<float> v;
    v.r = a.r; v.q = a.q; v.p = a.p; v.y = a.e;
    v.E = a.cs[0]; v.N = a.cs[1]; v.U = a.cs[2]; v.d = a.d;
    v.n = (int)N; v.nI = (int)A.nI; v.nIJ = (int)A.nIJ;
    if (a.project) project_mean(grid, const_cast<double*>(a.b), N, t0, T);
    double bb;
    {
        double s[1] = {0.}, t[1];
        for (long long c = t0; c < N; c += T) {
            const double bv = a.b[c], rs = sg * a.S[c] * bv;
            v.r[c] = (float)rs; v.q[c] = 0.f; v.p[c] = 0.f; v.y[c] = 0.f;
            a.x[c] = 0.;
            s[0] += bv * bv;
        }
        grid.sum<1>(s, t);
        bb = t[0];
    }
    MxWatch watch;
    watch.tol2 = fmax(a.rtol * a.rtol * bb, a.atol * a.atol);
    watch.start(bb);
    int it = 0, outer = 0, status = 0;
    double relres = bb > 0. ? 1. : 0., alpha = 0., beta = 0.;
    bool done = !(bb > 0.) || bb <= watch.tol2;
    if (bb != bb) status = 3;
    if (!scaled_form(a.out)) { done = true; status = 2; }   // not a definite symmetric system: the FP64 solve takes it
    bool fresh = true;   // the next update forms p = r + beta p only
    while (!done) {
        double acc[4] = {0., 0., 0., 0.}, tot[4];
        cg_update<float, W>(v, (float)alpha, (float)beta, false, acc[0], acc[1]);
        grid.sync();
        cg_product<float, W>(v, true, acc[2], acc[3]);
        grid.sum<4>(acc, tot);
        if (!fresh) ++it;
        const bool broke = !cg_scalars(tot[0], tot[2], tot[3], alpha, beta), stuck = broke && fresh;
        const bool due = (!fresh && watch.due(tot[1])) || tot[1] != tot[1];
        fresh = false;
        if (due || broke || it >= a.maxit) {
            // ---- x += S y; FP64 true residual in the place of the recursive one; p and q stay
            for (long long c = t0; c < N; c += T) { a.x[c] = a.x[c] + a.S[c] * (double)v.y[c]; v.y[c] = 0.f; }
            grid.sync();
            double s[2] = {0., 0.}, t[2];
            for (long long c = t0; c < N; c += T) {
                double y[1];
                apply<1>(A, c, [&](int, long long e) { return a.x[e]; }, y);
                const double rt = a.b[c] - y[0], rs = sg * a.S[c] * rt;
                v.r[c] = (float)rs;
                s[0] += rt * rt; s[1] += rs * rs;
            }
            grid.sum<2>(s, t);
            ++outer;
            relres = sqrt(t[0] / bb);
            if (t[0] <= watch.tol2) { done = true; status = 0; }
            else if (t[0] != t[0]) { done = true; status = 3; }
            else if (it >= a.maxit) { done = true; status = 1; }
            else {
                const bool restart = watch.refine(tot[1], t[0]) || broke;
                if (watch.stalls >= 2 || stuck) { done = true; status = 2; }
                if (restart || !cg_scalars(t[1], tot[2], tot[3], alpha, beta)) { alpha = beta = 0.; fresh = true; }
            }
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out->iters[0] = it; a.out->iters[1] = outer; a.out->relres[0] = relres; a.out->status[0] = status;
    }
}

// ------------------------------------------------------------------ host side
int sm_count() {
    static PerDevice<int> count;
    const int dev = current_device();
    return count.get(dev, [&] {
        int n = 0;
        return cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0 ? n : 148;
    });
}

// Shape of a persistent launch over n work items (one per thread and step of the sweep): as many
// threads per block, a power of two from 128, as give every item a thread of its own on all SMs, up to
// what the kernel's registers allow; past that the sweep takes several steps.  Fewer, fuller blocks make
// the reduction cheaper (1.5 us on 8 blocks, 2.4 on 148), but the loads of a sweep want every SM: CG
// per iteration, us, blocks of 512 and up against this rule: 34x32x32 7.4 and 5.7, 44x40x38 7.9 and
// 5.7, 56x50x48 8.0 and 6.4, 101x67x53 10.3 both.
template <auto Kernel>
static int launch_coop(long long n, void** params, cudaStream_t st) {
    static const int maxThreads = [] {
        cudaFuncAttributes f;
        return cudaFuncGetAttributes(&f, (const void*)Kernel) == cudaSuccess ? std::min(f.maxThreadsPerBlock, GR_THREADS) : 256;
    }();
    const int nsm = sm_count();
    int block = 128;
    while (block < maxThreads && n > (long long)block * nsm) block = std::min(2 * block, maxThreads);
    const int grid = (int)std::min<long long>(nsm, (n + block - 1) / block);
    CB_CUDA(cudaLaunchCooperativeKernel((const void*)Kernel, dim3(grid), dim3(block), params, 0, st));
    return 0;
}
template <auto Kernel, class Op>
static int launch_coop(const Op& op, KArgs& args, cudaStream_t st) {
    void* params[2] = {const_cast<Op*>(&op), &args};
    return launch_coop<Kernel>(args.N, params, st);
}

size_t krylov_partial_doubles() { return std::max(gr_doubles(sm_count()), gr_ordered_doubles(KB_PER_SM * sm_count())); }

template <class Op>
static int prepare(const Op& A, const Lat& L, const KspWork& w, cudaStream_t st) {
    inv_diag_kernel<Op><<<grid_for(L.N, 256), 256, 0, st>>>(A, L.N, w.invD, w.partials);
    CB_CHECK_LAUNCH();
    return 0;
}

static KArgs make_args(const Lat& L, const KspWork& w, const double* b, double* x, double rtol, int maxit, double atol) {
    KArgs a;
    a.b = b; a.x = x; a.r = w.r; a.rp = w.rp; a.s = w.r + L.PS;
    a.p[0] = w.p[0]; a.p[1] = w.p[1]; a.v[0] = w.v[0]; a.v[1] = w.v[1];
    a.t = w.t; a.invD = w.invD; a.partials = w.partials; a.out = w.out;
    a.N = L.N; a.PS = L.PS; a.rtol = rtol; a.atol = atol; a.maxit = maxit;
    a.project = 0;
    a.skip_if_ok = nullptr;
    a.fallbacks = nullptr;
    for (int q = 0; q < 3; ++q) a.cs[q] = w.cs[q];
    return a;
}

// The two CG launches: the scaled form, and the general one for the systems it does not take
// (each returns at once where the other runs).  Groups of two cells where the rows are even.
template <class Op>
static int run_cg(const Op& A, const Lat& L, const KspWork& w, KArgs& a, cudaStream_t st) {
    if (w.cs[0] && L.N < (1ll << 31) - 2 * L.nIJ) {
        CB_CUDA(cudaMemsetAsync(&w.out->general, 0, sizeof(int), st));
        scale_kernel<Op, double><<<grid_for(L.N, 256), 256, 0, st>>>(A, L.N, w.invD, w.cs[0], w.cs[1], w.cs[2], &w.out->general, w.partials);
        CB_CHECK_LAUNCH();
        auto al = [](const void* p) { return ((uintptr_t)p & 15u) == 0; };
        const bool v2 = L.nI % 2 == 0 && al(a.r) && al(a.v[0]) && al(a.p[0]) && al(a.x) &&
                        al(a.cs[0]) && al(a.cs[1]) && al(a.cs[2]) && al(diag_plane(A));
        void* params[2] = {const_cast<Op*>(&A), &a};
        if (v2 ? launch_coop<cgs_kernel<Op, 2>>(L.N / 2, params, st) : launch_coop<cgs_kernel<Op, 1>>(L.N, params, st)) return 1;
    } else
        for (int q = 0; q < 3; ++q) a.cs[q] = nullptr;
    if (prepare(A, L, w, st)) return 1;
    return launch_coop<cg1_kernel<Op>>(A, a, st);
}

int ksp_bicgstab(const Op7& A, int nr, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit,
                 cudaStream_t st, double atol) {
    if (ksp_small_fits(L)) return ksp_small(A, false, nr, b, x, L, w, rtol, maxit, st, 0, atol);
    if (prepare(A, L, w, st)) return 1;
    KArgs a = make_args(L, w, b, x, rtol, maxit, atol);
    if (nr == 3) {
        void* params[2] = {const_cast<Op7*>(&A), &a};
        CB_CUDA(cudaLaunchCooperativeKernel((const void*)bicgstab3_kernel<3, Op7>, dim3(KB_PER_SM * sm_count()), dim3(KB), params, 0, st));
        return 0;
    }
    return launch_coop<bicgstab_kernel<Op7>>(A, a, st);
}

int ksp_bicgstab_sym(const OpSym& A, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit,
                     cudaStream_t st, int project, double atol) {
    if (ksp_small_fits(L)) return ksp_small(A, false, b, x, L, w, rtol, maxit, st, project, atol, nullptr, nullptr);
    if (prepare(A, L, w, st)) return 1;
    KArgs a = make_args(L, w, b, x, rtol, maxit, atol);
    a.project = project;
    return launch_coop<bicgstab_kernel<OpSym>>(A, a, st);
}

int ksp_cg(const OpSym& A, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit, cudaStream_t st,
           int project, double atol) {
    if (ksp_small_fits(L)) return ksp_small(A, true, b, x, L, w, rtol, maxit, st, project, atol, nullptr, nullptr);
    KArgs a = make_args(L, w, b, x, rtol, maxit, atol);
    a.project = project;
    return run_cg(A, L, w, a, st);
}

int ksp_cg7(const Op7& A, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit, cudaStream_t st,
            double atol) {
    if (ksp_small_fits(L)) return ksp_small(A, true, 1, b, x, L, w, rtol, maxit, st, 0, atol);
    KArgs a = make_args(L, w, b, x, rtol, maxit, atol);
    return run_cg(A, L, w, a, st);
}

int ksp_csr(const OpCSR& A, int method, long long n, int longest, const double* b, double* x, const KspWork& w, double rtol, int maxit,
            cudaStream_t st, double atol) {
    Lat L;
    std::memset(&L, 0, sizeof(L));
    L.nI = (int)n; L.nJ = 1; L.nK = 1; L.N = n; L.nIJ = n; L.H = 0; L.PS = n;   // unpadded vectors
    if (ksp_small_fits_csr(n, longest)) return ksp_small(A, method == CAFFE_KSP_CG_JACOBI_INT, b, x, L, w, rtol, maxit, st, atol);
    if (prepare(A, L, w, st)) return 1;
    KArgs a = make_args(L, w, b, x, rtol, maxit, atol);
    for (int q = 0; q < 3; ++q) a.cs[q] = nullptr;
    return method == CAFFE_KSP_CG_JACOBI_INT ? launch_coop<cg1_kernel<OpCSR>>(A, a, st) : launch_coop<bicgstab_kernel<OpCSR>>(A, a, st);
}

int ksp_mixed_sym(const OpSym& A, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit,
                  cudaStream_t st, int project, double atol) {
    MxArgs m;
    m.b = b; m.x = x;
    m.r = w.fr; m.q = w.fq; m.p = w.fp; m.e = w.fe; m.d = w.fd; m.S = w.invD;
    for (int q = 0; q < 3; ++q) m.cs[q] = w.fB[q];
    m.partials = w.partials; m.out = w.out; m.N = L.N; m.rtol = rtol; m.atol = atol; m.maxit = maxit; m.project = project;
    CB_CUDA(cudaMemsetAsync(&w.out->general, 0, sizeof(int), st));
    cast_kernel<<<grid_for(L.N, 256), 256, 0, st>>>(L.N, A.aP, w.fd);
    scale_kernel<OpSym, float><<<grid_for(L.N, 256), 256, 0, st>>>(A, L.N, w.invD, w.fB[0], w.fB[1], w.fB[2], &w.out->general, w.partials);
    CB_CHECK_LAUNCH();
    void* params[2] = {const_cast<OpSym*>(&A), &m};
    // cell arrays start 16-byte aligned; groups of 16 bytes where the rows are multiples of them
    return L.nI % 4 == 0 ? launch_coop<mixed_cg_kernel<4>>(L.N / 4, params, st) : launch_coop<mixed_cg_kernel<1>>(L.N, params, st);
}

int ksp_fallback_sym(const OpSym& A, int method, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit,
                     cudaStream_t st, int project, const int* status, int* fallbacks, double atol) {
    // plain FP64 re-solve from zero, executed only when *status (the previous solve's) is non-zero
    if (ksp_small_fits(L))
        return ksp_small(A, method == CAFFE_KSP_CG_JACOBI_INT, b, x, L, w, rtol, maxit, st, project, atol, status, fallbacks);
    KArgs a = make_args(L, w, b, x, rtol, maxit, atol);
    a.project = project;
    a.skip_if_ok = status;
    a.fallbacks = fallbacks;
    if (method == CAFFE_KSP_CG_JACOBI_INT) return run_cg(A, L, w, a, st);
    if (prepare(A, L, w, st)) return 1;
    return launch_coop<bicgstab_kernel<OpSym>>(A, a, st);
}

}  // namespace cb
