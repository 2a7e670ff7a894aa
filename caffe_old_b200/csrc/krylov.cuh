// Krylov solvers on the device: operators, workspace and launchers.
#pragma once
#include "common.cuh"

namespace cb {

// Immersed-boundary ghost rows in ELL-9 form, sorted by cell (IbPiso.cpp:119-190):
// col[9g + 0] is the ghost cell itself, col[9g + 1..8] the interpolation stencil (-1 for a
// dropped column), val[9g + m] the coefficients; words has one
// entry per 32 cells: a bit per ghost cell, and the number of ghost cells before them.
struct GhostRows {
    int n;
    const int* cell;
    const int* col;
    const double* val;
    const uint2* words;
};

// Non-symmetric 7-point operator: 7 per-cell coefficient arrays (momentum, Simple.cpp:162-171).
struct Op7 {
    const double* a[7];
    long long nI, nIJ;
    GhostRows gh;
};

// Symmetric 7-point operator: diagonal plus east/north/top coefficients per cell; the
// west/south/bottom coefficient of a cell is the east/north/top one of that neighbour
// (pressure correction, Simple.cpp:241-265).
struct OpSym {
    const double* aP;
    const double* aE;
    const double* aN;
    const double* aT;
    long long nI, nIJ;
    GhostRows gh;
};

// General sparse operator in compressed rows: the AIJ matrix SparseMatrix assembles row by row
// (src/Math/SparseMatrix.cpp:49-83).  diag[r] is the position of row r's diagonal entry in
// col / val, -1 when the row has none.
struct OpCSR {
    const int* ptr;
    const int* col;
    const double* val;
    const int* diag;
};

struct KspOut {
    int iters[3];
    double relres[3];
    int status[3];      // 0 converged, 1 maxit, 2 breakdown, 3 non-finite
    int cascades;       // learned solve only: 1 when its network stage handed over to the pyramid stage
    int general;        // CG: set when the scaled form does not apply to the system
    int net_iters;      // learned solve only: inner iterations run with the network in the preconditioner
};

// Workspace for up to NR = 3 right-hand sides; every array is a halo-padded cell array of
// 3 planes (a single right-hand side also uses the plane after r as a second buffer).
struct KspWork {
    double* r;
    double* rp;
    double* p[2];
    double* v[2];
    double* t;
    double* invD;     // one plane
    double* cs[3];    // CG: off-diagonal planes of the scaled operator (null: the unscaled form runs)
    double* partials; // slots of the grid reductions: krylov_partial_doubles()
    KspOut* out;      // device
    // single-precision workspace of the mixed-precision solver (halo-padded float cell arrays)
    float *fr, *fq, *fp, *fe;
    float* fd;        // diagonal
    float* fB[3];     // off-diagonal planes of the scaled operator
};

// Every solve stops once ||b - A x|| <= max(rtol ||b||, atol) in the FP64 true residual (the
// convergence test of PETSc's KSP, rtol and atol; atol = 0 leaves the relative test alone).
int ksp_bicgstab(const Op7& A, int nr, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit,
                 cudaStream_t st, double atol = 0.);
// project != 0: remove the mean of b first (b is modified), for singular all-Neumann systems
int ksp_bicgstab_sym(const OpSym& A, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit,
                     cudaStream_t st, int project = 0, double atol = 0.);
int ksp_cg(const OpSym& A, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit, cudaStream_t st,
           int project = 0, double atol = 0.);
int ksp_cg7(const Op7& A, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit, cudaStream_t st,
            double atol = 0.);
// FP64 iterative refinement around FP32 CG on the symmetric p' operator (no ghost rows).
// out->iters[0] counts the FP32 iterations, iters[1] the refinements.
int ksp_mixed_sym(const OpSym& A, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit,
                  cudaStream_t st, int project, double atol = 0.);
// Plain FP64 re-solve that runs only when *status is non-zero (the fallback of a mixed or
// learned solve), decided on the device without a host round trip.
int ksp_fallback_sym(const OpSym& A, int method, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit,
                     cudaStream_t st, int project, const int* status, int* fallbacks, double atol = 0.);
// Krylov solve of an n-row compressed-row system (vectors of n doubles, no halo): BiCGStab or CG
// with Jacobi preconditioning, the same persistent kernels as the lattice solves; longest: entries of
// the longest row.
int ksp_csr(const OpCSR& A, int method, long long n, int longest, const double* b, double* x, const KspWork& w, double rtol, int maxit,
            cudaStream_t st, double atol = 0.);
// The same solves inside one thread-block cluster, for systems whose vectors fit its registers and
// shared memory (krylov_small.cu).  rhs right-hand sides PS apart, each solved by a cluster of its own.
bool ksp_small_fits(const Lat& L);
bool ksp_small_fits_csr(long long n, int longest);
int ksp_small(const Op7& A, bool cgMethod, int rhs, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit,
              cudaStream_t st, int project, double atol);
int ksp_small(const OpSym& A, bool cgMethod, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit, cudaStream_t st,
              int project, double atol, const int* skip_if_ok, int* fallbacks);
int ksp_small(const OpCSR& A, bool cgMethod, const double* b, double* x, const Lat& L, const KspWork& w, double rtol, int maxit, cudaStream_t st,
              double atol);
// Doubles of slot memory (KspWork::partials) that the reductions of a solve take on this device.
size_t krylov_partial_doubles();

}  // namespace cb
