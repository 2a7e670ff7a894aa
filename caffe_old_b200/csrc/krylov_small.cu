// Krylov solves of small systems inside one thread-block cluster.
//
// A solve on a lattice of a few thousand cells is a chain of latencies: on the whole grid an iteration
// of the 64x64 SIMPLE cavity took 8.2 us, of which moving its 4096 cells is nothing.  Here
// one cluster of up to 16 blocks holds the whole solve on chip: the operator's seven planes,
// the vector it is applied to (with a halo that the neighbouring blocks write), x, 1/d and BiCGStab's
// shadow residual in shared memory, the other vectors in registers, one to four cells per
// thread.  Barriers and sums run over the cluster's own barrier, about 0.3 and 0.8 us against
// 1.6 and 2.6 us for the grid's.  Right-hand sides are solved by clusters of their own, side by side.
//
// Measured (us per iteration, grid -> cluster): BiCGStab 64x64 8.2 -> 3.7, 210x130
// 9.8 -> 7.4; CG 28x24x20 5.7 -> 3.3.  FP32 CG takes 5.5 on the 64x64 case: the mixed form runs here too.
//
// The methods are those of krylov.cu (right-preconditioned BiCGStab, Jacobi-CG, both with merged
// reductions and the true-residual stopping test); CG here keeps the unscaled operator, so that it takes
// every system the general form takes.
#include <algorithm>
#include <cooperative_groups.h>
#include <cstring>
#include <type_traits>

#include "bicgstab.cuh"
#include "cg_scaled.cuh"
#include "gridred.cuh"
#include "krylov.cuh"
#include "perdevice.h"
#include "stencil.cuh"

namespace cg = cooperative_groups;

namespace cb {
namespace {

constexpr int S_THREADS = 512;     // threads per block at most
constexpr int S_BLOCKS = 16;       // blocks of a cluster at most
constexpr int S_CELLS = 4;         // cells per thread at most
constexpr int S_VECS = 4;          // planes in shared memory beside the operator's: ex, x, 1/d, shadow residual

constexpr int S_BYTES = 216 * 1024;   // dynamic shared memory of a block at most

struct SmallArgs {
    double* b;
    double* x;
    KspOut* out;
    long long N, PS;
    int shift;          // a block's cells: 1 << shift
    int halo;           // cells before and after a block's that its rows reach
    double rtol, atol;
    int maxit;
    int project;
    const int* skip_if_ok;
    int* fallbacks;
};

// Sums over the cluster, the same bits in every thread.
template <int SB>
struct ClusterSum {
    int parity = 0;
    template <int K>
    __device__ __forceinline__ void operator()(cg::cluster_group& cl, const double (&v)[K], double (&out)[K]) {
        static_assert(K <= 8, "values of one sum");
        __shared__ double sm[SB / 32][8];
        __shared__ double inbox[2][S_BLOCKS][8];
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, R = (int)cl.num_blocks(), me = (int)cl.block_rank();
        const double c = gr_warp_sums(v, lane);
        if (lane < 8) sm[w][lane] = c;
        __syncthreads();
        if (w == 0) {
            double t = 0.;
#pragma unroll
            for (int u = 0; u < SB / 128; ++u) t += sm[(lane >> 3) + 4 * u][lane & 7];
            t += __shfl_xor_sync(0xffffffffu, t, 8);
            t += __shfl_xor_sync(0xffffffffu, t, 16);
            if ((lane & 7) < K)
                for (int r = lane >> 3; r < R; r += 4) *cl.map_shared_rank(&inbox[parity][me][lane & 7], r) = t;
        }
        cl.sync();
        double x[K];
#pragma unroll
        for (int q = 0; q < K; ++q) x[q] = lane < R ? inbox[parity][lane][q] : 0.;
        const double d = gr_warp_sums(x, lane);
#pragma unroll
        for (int q = 0; q < K; ++q) out[q] = __shfl_sync(0xffffffffu, d, q);
        parity ^= 1;   // this buffer is written again two barriers on, when every block has read it
    }
};

// The vector the operator is applied to, spread over the cluster's blocks: ex[0 .. len) are this
// block's cells, with `halo` cells of the neighbouring blocks before and after.  A block writes its cells
// into every halo that holds them (a store needs no answer; the barrier that follows orders it), so
// that a row reads this block's memory only.
struct Spread {
    double* ex;
    int shift, halo, me, last, base, len;   // this block's cells: [base, base + len)
    __device__ __forceinline__ void put(cg::cluster_group& cl, int l, double v) const {
        const int c = base + l;
        ex[l] = v;
        for (int r = max(c - halo, 0) >> shift; r <= min((c + halo) >> shift, last); ++r)
            if (r != me) *cl.map_shared_rank(ex + (c - (r << shift)), r) = v;
    }
    // any cell of the lattice
    __device__ __forceinline__ double at(cg::cluster_group& cl, int g) const {
        const int r = g >> shift;
        return *cl.map_shared_rank(ex + (g - (r << shift)), r);
    }
    __device__ __forceinline__ uint32_t address(int g) const {
        const int r = g >> shift;
        uint32_t a = (uint32_t)__cvta_generic_to_shared(ex + (g - (r << shift)));
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(a), "r"(r));
        return a;
    }
};

// Operators on the cluster: the seven planes of a thread's cells in registers, or, with more than two
// cells per thread, in shared memory (a product's 14 shared-memory reads per cell are what bounds
// a sweep once a block holds a thousand cells).
template <class Op, int C, int SB>
struct SmallOp {
    static constexpr bool inRegs = C <= 2;
    Op A;
    double k[inRegs ? 7 : 1][inRegs ? C : 1];
    double* co;   // [7][1 << shift]
    int nI, nIJ;
    __device__ __forceinline__ void load(cg::cluster_group&, const Op& op, double* mem, const Spread& s, double* id) {
        A = op; co = mem; nI = (int)op.nI; nIJ = (int)op.nIJ;
#pragma unroll
        for (int m = 0; m < C; ++m) {
            const int l = (int)threadIdx.x + SB * m;
            double a[7] = {0., 0., 0., 0., 0., 0., 0.};
            if (l < s.len) {
                planes(op, s.base + l, a);
                id[l] = a[0] != 0. ? 1. / a[0] : 1.;
            }
#pragma unroll
            for (int q = 0; q < 7; ++q) {
                if (inRegs) k[inRegs ? q : 0][inRegs ? m : 0] = a[q];
                else if (l < s.len) co[(q << s.shift) + l] = a[q];
            }
        }
    }
    static __device__ __forceinline__ void planes(const Op7& op, long long c, double (&a)[7]) {
#pragma unroll
        for (int q = 0; q < 7; ++q) a[q] = op.a[q][c];
    }
    static __device__ __forceinline__ void planes(const OpSym& op, long long c, double (&a)[7]) {
        a[0] = op.aP[c]; a[1] = op.aE[c]; a[2] = op.aE[c - 1]; a[3] = op.aN[c]; a[4] = op.aN[c - op.nI];
        a[5] = op.aT[c]; a[6] = op.aT[c - op.nIJ];
    }
    // row of slot m, cell l of the block; a neighbour beyond the lattice's ends has coefficient zero,
    // and the halo there is never written (zero)
    __device__ __forceinline__ double row(cg::cluster_group& cl, const Spread& s, int m, int l) const {
        const int c = s.base + l;
        const double* x = s.ex + l;
        auto a = [&](int q) { return inRegs ? k[inRegs ? q : 0][inRegs ? m : 0] : co[(q << s.shift) + l]; };
        double y = a(0) * x[0] + a(1) * x[1] + a(2) * x[-1];
        if (s.halo >= nI) y += a(3) * x[nI] + a(4) * x[-nI];
        if (s.halo >= nIJ) y += a(5) * x[nIJ] + a(6) * x[-nIJ];
        if (A.gh.n > 0) {
            const uint2 w = __ldg(A.gh.words + (c >> 5));
            double t[1];
            if (is_ghost(w, c)) {
                ghost_row<1>(A.gh, ghost_index(w, c), [&](int, long long e) { return s.at(cl, (int)e); }, t);
                y = t[0];
            }
        }
        return y;
    }
    static constexpr int planesOf = inRegs ? 0 : 7;
};
// Compressed rows: the first E entries of a thread's rows are kept in registers, each as its value and the
// place of its column's cell in the cluster, so that a product is E independent shared-memory reads in
// place of a chain through global memory (row bounds, then column, then the cell).  E = 8 covers the 5- and
// 7-point rows; longer rows read the rest as before.  us per BiCGStab iteration on 5-point rows: 6300
// rows 6.7 -> 4.4, 12000 7.9 -> 5.9.
template <int C, int SB>
struct SmallOp<OpCSR, C, SB> {
    static constexpr int E = 8;
    OpCSR A;
    int p0[C], p1[C];
    double val[C][E];
    uint32_t src[C][E];   // shared-memory addresses in the cluster's window
    __device__ __forceinline__ void load(cg::cluster_group& cl, const OpCSR& op, double*, const Spread& s, double* id) {
        A = op;
#pragma unroll
        for (int m = 0; m < C; ++m) {
            const int l = (int)threadIdx.x + SB * m, c = s.base + l;
            p0[m] = p1[m] = 0;
            if (l < s.len) {
                const double d = diag_of(A, c);
                id[l] = d != 0. ? 1. / d : 1.;
                p0[m] = __ldg(A.ptr + c); p1[m] = __ldg(A.ptr + c + 1);
            }
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const bool has = p0[m] + e < p1[m];
                val[m][e] = has ? __ldg(A.val + p0[m] + e) : 0.;
                src[m][e] = s.address(has ? __ldg(A.col + p0[m] + e) : s.base);
            }
        }
    }
    __device__ __forceinline__ double row(cg::cluster_group& cl, const Spread& s, int m, int) const {
        double x[E], y = 0.;
#pragma unroll
        for (int e = 0; e < E; ++e) asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(x[e]) : "r"(src[m][e]) : "memory");
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (p0[m] + e < p1[m]) y += val[m][e] * x[e];
#pragma unroll 1
        for (int p = p0[m] + E; p < p1[m]; ++p) y += __ldg(A.val + p) * s.at(cl, __ldg(A.col + p));
        return y;
    }
    static constexpr int planesOf = 0;
};

// What both methods share: the block's place, the right-hand side (projected if asked), its norm.
template <class Op, int C, int SB>
struct Frame {
    cg::cluster_group cl;
    Spread s;
    SmallOp<Op, C, SB> A;
    ClusterSum<SB> sum;
    double *b, *x, *id, *rp;    // b in global memory; x, 1/d and the shadow residual in shared memory
    double* xOut;
    double bb, tol2, relres = 0.;
    int it = 0, status = 0;
    bool done;

    __device__ Frame(const Op& op, const SmallArgs& a, double* mem, int rhs) : cl(cg::this_cluster()) {
        s.shift = a.shift; s.me = (int)cl.block_rank(); s.base = s.me << a.shift;
        s.len = (int)max(0ll, min((long long)1 << a.shift, a.N - s.base));
        s.halo = a.halo; s.last = (int)cl.num_blocks() - 1;
        s.ex = mem + a.halo;
        mem += 2 * a.halo;
        x = mem + (1 << a.shift); id = mem + (2 << a.shift); rp = mem + (3 << a.shift);
        for (int l = (int)threadIdx.x - a.halo; l < (1 << a.shift) + a.halo; l += SB) s.ex[l] = 0.;
        A.load(cl, op, mem + (S_VECS << a.shift), s, id);
        b = a.b + rhs * a.PS + s.base; xOut = a.x + rhs * a.PS + s.base;
        __syncthreads();
        each([&](int, int l) { x[l] = 0.; });
        cl.sync();   // every block runs before its shared memory is written from outside
        double t[1];
        if (a.project)   // twice: see project_mean in krylov.cu
            for (int pass = 0; pass < 2; ++pass) {
                double m[1] = {0.};
                each([&](int, int l) { m[0] += b[l]; });
                sum(cl, m, t);
                const double mean = t[0] / (double)a.N;
                each([&](int, int l) { b[l] = b[l] - mean; });
            }
        double v[1] = {0.};
        each([&](int, int l) { rp[l] = b[l]; v[0] += b[l] * b[l]; });
        sum(cl, v, t);
        bb = t[0];
        tol2 = fmax(a.rtol * a.rtol * bb, a.atol * a.atol);
        done = !(bb > 0.) || bb <= tol2;   // x = 0 already meets the absolute floor
        if (bb > 0. && done) relres = 1.;
        if (bb != bb) status = 3;
    }
    // f(k, l) for the thread's cells: slot k, cell l of the block
    template <class F>
    __device__ __forceinline__ void each(F&& f) const {
#pragma unroll
        for (int k = 0; k < C; ++k) {
            const int l = (int)threadIdx.x + SB * k;
            if (l < s.len) f(k, l);
        }
    }
    // true residual of x into r; decides.  Every thread of the cluster calls it.
    __device__ void check(double (&r)[C], int maxit, double& rr) {
        each([&](int, int l) { s.put(cl, l, x[l]); });
        cl.sync();
        double v[1] = {0.}, t[1];
        each([&](int k, int l) { r[k] = b[l] - A.row(cl, s, k, l); v[0] += r[k] * r[k]; });
        sum(cl, v, t);
        rr = t[0];
        relres = sqrt(rr / bb);
        if (rr <= tol2) { done = true; status = 0; }
        else if (rr != rr) { done = true; status = 3; }
        else if (it >= maxit) { done = true; status = 1; }
    }
    __device__ void finish(KspOut* out, int rhs) {
        each([&](int, int l) { xOut[l] = x[l]; });
        if (s.me == 0 && threadIdx.x == 0) { out->iters[rhs] = it; out->relres[rhs] = relres; out->status[rhs] = status; }
        cl.sync();   // no block leaves while another may read its shared memory
    }
};

__device__ __forceinline__ bool skipped(const SmallArgs& a) {
    if (!a.skip_if_ok) return false;
    if (*a.skip_if_ok == 0) return true;
    if (blockIdx.x == 0 && threadIdx.x == 0 && a.fallbacks) atomicAdd(a.fallbacks, 1);
    return false;
}

template <class Op, int C, int SB>
__global__ void __launch_bounds__(SB) small_bicgstab_kernel(Op op, SmallArgs a) {
    extern __shared__ double small_mem[];
    if (skipped(a)) return;   // uniform across the grid
    const int rhs = blockIdx.y;
    Frame<Op, C, SB> f(op, a, small_mem, rhs);
    double r[C], p[C], v[C], t[C];
#pragma unroll
    for (int k = 0; k < C; ++k) r[k] = p[k] = v[k] = t[k] = 0.;
    f.each([&](int k, int l) { r[k] = f.b[l]; });
    double rho = f.bb, rp2 = f.bb, alpha = 0., omega = 0., beta = 0.;
    while (!f.done) {
        f.each([&](int k, int l) { p[k] = r[k] + beta * (p[k] - omega * v[k]); f.s.put(f.cl, l, f.id[l] * p[k]); });
        f.cl.sync();
        double s1[1] = {0.}, rv[1];
        f.each([&](int k, int l) { v[k] = f.A.row(f.cl, f.s, k, l); s1[0] += f.rp[l] * v[k]; });
        f.sum(f.cl, s1, rv);
        bool check = rv[0] == 0. || rv[0] != rv[0];
        if (!check) {
            alpha = rho / rv[0];
            f.each([&](int k, int l) { r[k] = r[k] - alpha * v[k]; f.s.put(f.cl, l, f.id[l] * r[k]); });   // s
            f.cl.sync();
            double s5[5] = {0., 0., 0., 0., 0.}, d[5];
            f.each([&](int k, int l) {
                t[k] = f.A.row(f.cl, f.s, k, l);
                s5[0] += t[k] * r[k]; s5[1] += t[k] * t[k];
                s5[2] += f.rp[l] * r[k]; s5[3] += f.rp[l] * t[k];
                s5[4] += r[k] * r[k];
            });
            f.sum(f.cl, s5, d);
            f.it += 1;
            omega = d[1] == 0. ? 0. : d[0] / d[1];
            f.each([&](int k, int l) {
                f.x[l] = f.x[l] + (alpha * (f.id[l] * p[k]) + omega * f.s.ex[l]);
                r[k] = r[k] - omega * t[k];
            });
            const double rn = d[2] - omega * d[3], rr = d[4] - 2. * omega * d[0] + omega * omega * d[1];
            beta = (rn / rho) * (alpha / omega);
            rho = rn;
            check = rr <= f.tol2 || omega == 0. || f.it >= a.maxit || rr != rr || !bi_sound(rn, rp2, rr);
        } else
            f.it += 1;   // a breakdown counts: from the same residual it repeats, and maxit must end it
        if (check) {
            double rr;
            f.check(r, a.maxit, rr);
            // a restart from the true residual, if the solve goes on
            f.each([&](int k, int l) { f.rp[l] = r[k]; p[k] = v[k] = 0.; });
            rho = rp2 = rr; alpha = omega = beta = 0.;
        }
    }
    f.finish(a.out, rhs);
}

// Jacobi-CG with one reduction per iteration (cg_scaled.cuh), z = D^-1 r:
//   r -= alpha q;  p = z + beta p;  x += alpha p_old;  q = A p;  sums (r, z), (r, r), (p, q), (q, D^-1 q)
template <class Op, int C, int SB>
__global__ void __launch_bounds__(SB) small_cg_kernel(Op op, SmallArgs a) {
    extern __shared__ double small_mem[];
    if (skipped(a)) return;   // uniform across the grid
    Frame<Op, C, SB> f(op, a, small_mem, 0);
    double r[C], p[C], q[C];
#pragma unroll
    for (int k = 0; k < C; ++k) r[k] = p[k] = q[k] = 0.;
    f.each([&](int k, int l) { r[k] = f.b[l]; });
    const double growth = a.project ? CG_GROWTH : 1e300;   // NaN counts as growth
    double alpha = 0., beta = 0., best = f.bb;
    bool first = true;
    while (!f.done) {
        double s4[4] = {0., 0., 0., 0.}, d[4];
        f.each([&](int k, int l) {
            r[k] = r[k] - alpha * q[k];
            f.x[l] = f.x[l] + alpha * p[k];
            const double z = f.id[l] * r[k];
            p[k] = z + beta * p[k];
            f.s.put(f.cl, l, p[k]);
            s4[0] += r[k] * z; s4[1] += r[k] * r[k];
        });
        f.cl.sync();
        f.each([&](int k, int l) {
            q[k] = f.A.row(f.cl, f.s, k, l);
            s4[2] += p[k] * q[k]; s4[3] += q[k] * (f.id[l] * q[k]);
        });
        f.sum(f.cl, s4, d);
        if (!first) f.it += 1;
        alpha = d[0] / d[2];
        beta = (alpha * alpha * d[3] - d[0]) / d[0];   // negative where (r, z) changes sign: 1/d need not be of one sign here
        const bool broke = d[0] == 0. || d[2] == 0. || alpha != alpha || beta != beta, stuck = broke && first;
        if (d[1] < best) best = d[1];
        if ((!first && (d[1] <= f.tol2 || f.it >= a.maxit)) || !(d[1] <= growth * best) || broke) {
            double rr;
            f.check(r, a.maxit, rr);
            if (!f.done && stuck) { f.done = true; f.status = 2; }   // no direction from a fresh residual
            // a restart from the true residual (in the range of a singular A), if the solve goes on
            alpha = beta = 0.; best = rr; first = true;
            f.each([&](int k, int) { p[k] = q[k] = 0.; });
            if (a.project && !f.done) {
                double m[1] = {0.}, tot[1];
                f.each([&](int k, int) { m[0] += r[k]; });
                f.sum(f.cl, m, tot);
                f.each([&](int k, int) { r[k] = r[k] - tot[0] / (double)a.N; });
            }
        } else
            first = false;
    }
    f.finish(a.out, 0);
}

size_t small_bytes(int planes, int shift, long long halo) { return sizeof(double) * (((size_t)(planes + S_VECS) << shift) + 2 * (size_t)halo); }

template <auto Kernel, int SB>
int launch_small(const void* op, SmallArgs& a, int rhs, int planes, int blocks, cudaStream_t st) {
    const size_t smem = small_bytes(planes, a.shift, a.halo);
    static PerDevice<bool> ready;
    if (!ready.get(current_device(), [] {
            return cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S_BYTES) == cudaSuccess &&
                   cudaFuncSetAttribute(Kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
        })) { set_error("small-system solve: kernel attributes refused"); return 1; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks, rhs);
    cfg.blockDim = dim3(SB);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = blocks; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    void* params[2] = {const_cast<void*>(op), &a};
    CB_CUDA(cudaLaunchKernelExC(&cfg, (const void*)Kernel, params));
    return 0;
}

// whether the current device runs a cluster of S_BLOCKS blocks of the largest form (asked once)
bool cluster_fits() {
    static PerDevice<bool> fits;
    return fits.get(current_device(), [] {
        auto k = small_bicgstab_kernel<Op7, S_CELLS, S_THREADS>;
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, S_BYTES) != cudaSuccess ||
            cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(S_BLOCKS);
        cfg.blockDim = dim3(S_THREADS);
        cfg.dynamicSmemBytes = S_BYTES;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = S_BLOCKS; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) { cudaGetLastError(); return false; }
        return n >= 1;
    });
}

// the fewest cells a block can hold with the whole cluster at work; at least a warp's
int shift_of(long long n) {
    int shift = 5;
    while (((long long)S_BLOCKS << shift) < n) ++shift;
    return shift;
}
// how far a row reaches (an extent of one has no neighbours)
long long halo_of(const Lat& L) { return L.nK > 1 ? L.nIJ : L.nJ > 1 ? L.nI : 1; }

template <class Op>
int run(const Op& A, bool cgMethod, int rhs, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit, cudaStream_t st,
        int project, double atol, const int* skip_if_ok, int* fallbacks) {
    SmallArgs a;
    a.b = const_cast<double*>(b); a.x = x; a.out = w.out; a.N = L.N; a.PS = L.PS;
    a.rtol = rtol; a.atol = atol; a.maxit = maxit; a.project = project; a.skip_if_ok = skip_if_ok; a.fallbacks = fallbacks;
    a.shift = shift_of(L.N);
    a.halo = (int)halo_of(L);
    const int blocks = (int)((L.N + (1ll << a.shift) - 1) >> a.shift);
    const int cells = 1 << a.shift;
#define SMALL_LAUNCH(C, SB)                                                                                                                  \
    return cgMethod ? launch_small<small_cg_kernel<Op, C, SB>, SB>(&A, a, rhs, SmallOp<Op, C, SB>::planesOf, blocks, st)                      \
                    : launch_small<small_bicgstab_kernel<Op, C, SB>, SB>(&A, a, rhs, SmallOp<Op, C, SB>::planesOf, blocks, st)
    // blocks of 256 threads where they hold their cells one each (64x64: 3.7 us an iteration against 4.3
    // with 512), else of 512
    if (cells <= 256) { SMALL_LAUNCH(1, 256); }
    if (cells <= 512) { SMALL_LAUNCH(1, 512); }
    if (cells <= 1024) { SMALL_LAUNCH(2, 512); }
    if constexpr (!std::is_same<Op, OpCSR>::value) { SMALL_LAUNCH(4, 512); }   // compressed rows: ksp_small_fits_csr
    set_error("small-system solve: too many rows");
    return 1;
#undef SMALL_LAUNCH
}

}  // namespace

bool ksp_small_fits(const Lat& L) {
    return L.N <= (long long)S_BLOCKS * S_THREADS * S_CELLS && small_bytes(7, shift_of(L.N), halo_of(L)) <= (size_t)S_BYTES && cluster_fits();
}

// Compressed rows: what lies beyond the registers is read entry by entry on 16 SMs, where the whole grid
// has nine times as many, so long rows and many rows per thread belong there.  us per BiCGStab
// iteration, cluster and grid, rows of 5 / 9 / 11 / 14 / 19 entries: 6000 rows 4.9 7.6 / 5.9 8.3 / 7.2 8.6 / 8.6 9.2 /
// 12.9 10.5; 12000 rows 6.9 8.0 / 8.6 8.7 / 11.1 8.9 / 13.1 10.1 / 21.8 10.7; 26000 rows, four per thread, 11.4
// 8.4 / 22.2 9.5 / 30.5 10.0 / 30.5 11.1 / 50.4 13.1.
bool ksp_small_fits_csr(long long n, int longest) {
    const bool one = n <= S_BLOCKS * S_THREADS, two = n <= 2 * S_BLOCKS * S_THREADS;   // rows per thread
    return ((one && longest <= 14) || (two && longest <= 9)) && cluster_fits();
}

int ksp_small(const Op7& A, bool cgMethod, int rhs, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit,
              cudaStream_t st, int project, double atol) {
    return run(A, cgMethod, rhs, b, x, L, w, rtol, maxit, st, project, atol, nullptr, nullptr);
}
int ksp_small(const OpSym& A, bool cgMethod, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit, cudaStream_t st,
              int project, double atol, const int* skip_if_ok, int* fallbacks) {
    return run(A, cgMethod, 1, b, x, L, w, rtol, maxit, st, project, atol, skip_if_ok, fallbacks);
}
int ksp_small(const OpCSR& A, bool cgMethod, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit, cudaStream_t st,
              double atol) {
    return run(A, cgMethod, 1, b, x, L, w, rtol, maxit, st, 0, atol, nullptr, nullptr);
}

}  // namespace cb
