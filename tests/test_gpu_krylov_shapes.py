"""The persistent Krylov kernels at the edges of their launch shapes and dispatch: one cell, the sizes
at which a cluster's blocks take more cells per thread or the system leaves the cluster (32768 cells, or
planes too large for a halo), rows too short or odd for the two-cell groups, one plane, sweeps of several steps, diagonals of either
sign, and the systems the scaled CG hands to the general one (mixed signs of the diagonal, a
matrix that is not symmetric).

Tolerance: the solve stops at a true relative residual of 1e-12, so the residual of the returned x,
evaluated on the host, is within 1e-11; on small systems x agrees with a dense solve to 1e-9 (condition
numbers up to about 1e3)."""
import numpy as np
import pytest

from caffe_old_b200 import _lib

from test_zz_no_alloc import seven_point_residual, seven_point_system

pytestmark = pytest.mark.gpu

RTOL = 1e-12


def dense(shape, coef):
    nI, nJ, _ = shape
    N = coef.shape[1]
    A = np.diag(coef[0])
    for q, off in ((1, 1), (3, nI), (5, nI * nJ)):
        for c in range(N - off):
            A[c, c + off] += coef[q][c]
            A[c + off, c] += coef[q + 1][c + off]
    return A


@pytest.mark.parametrize("sign", [-1.0, 1.0])
@pytest.mark.parametrize("method", ["cg_jacobi", "bicgstab_jacobi"])
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 1), (3, 1, 1), (1, 7, 2), (2, 2, 2), (33, 4, 3), (64, 3, 2), (64, 64, 1), (31, 13, 11), (25, 25, 25), (32, 32, 32), (33, 32, 32), (150, 150, 2),
                                   (129, 64, 33), (200, 120, 31)])
def test_solution_at_the_edges_of_the_launch_shapes(shape, method, sign):
    N = int(np.prod(shape))
    if N > 8:
        coef, b = seven_point_system(shape, 11, True)
    else:   # the generator wants a neighbour in every direction
        coef, b = np.zeros((7, N)), np.arange(1.0, N + 1.0)
        i, j, k = np.arange(N) % shape[0], (np.arange(N) // shape[0]) % shape[1], np.arange(N) // (shape[0] * shape[1])
        for q, inside in enumerate((i < shape[0] - 1, i > 0, j < shape[1] - 1, j > 0, k < shape[2] - 1, k > 0)):
            coef[q + 1][inside] = 1.0 + 0.1 * (q // 2)
        coef[0] = -coef[1:].sum(axis=0) - 0.15
    coef = sign * coef
    x, _, rr, st = _lib.ksp7_solve(shape, coef, b, method, RTOL, 20000)
    assert st == 0 and rr <= RTOL
    if N <= 500:
        ref = np.linalg.solve(dense(shape, coef), b)
        assert np.linalg.norm(x - ref) <= 1e-9 * np.linalg.norm(ref)
    else:
        assert seven_point_residual(shape, coef, x, b) <= 1e-11


def test_cg_on_a_diagonal_of_mixed_signs():
    shape = (6, 5, 4)
    rng = np.random.default_rng(3)
    coef = np.zeros((7, 120))
    coef[0] = rng.uniform(1.0, 2.0, 120) * np.where(np.arange(120) % 3 == 0, -1.0, 1.0)
    b = rng.standard_normal(120)
    x, _, _, st = _lib.ksp7_solve(shape, coef, b, "cg_jacobi", RTOL, 100)
    assert st == 0
    assert np.linalg.norm(x - b / coef[0]) <= 1e-11 * np.linalg.norm(x)


def test_cg_on_a_matrix_that_is_not_symmetric_runs_the_general_form():
    """Nearly symmetric: CG still converges, and only the operator as given leaves a small residual."""
    shape = (12, 9, 5)
    coef, b = seven_point_system(shape, 4, True)
    coef = coef.copy()
    coef[2] *= 1.0 + 1e-9
    x, _, rr, st = _lib.ksp7_solve(shape, coef, b, "cg_jacobi", RTOL, 5000)
    assert st == 0 and rr <= RTOL
    assert seven_point_residual(shape, coef, x, b) <= 1e-11


@pytest.mark.parametrize("n", [2, 32768, 40000])
@pytest.mark.parametrize("entry", ["ksp7", "csr"])
def test_bicgstab_breakdown_from_the_first_residual_ends_at_maxit(entry, n):
    """Pairs of cells with the matrix (0 1; -1 0) and b = 1: (r, A r) is zero exactly, from every restart."""
    even = np.arange(n) % 2 == 0
    b = np.ones(n)
    if entry == "ksp7":
        coef = np.zeros((7, n))
        coef[1][even], coef[2][~even] = 1.0, -1.0
        with pytest.raises(_lib.CaffeError):   # the call's answer to a solve that ends at maxit
            _lib.ksp7_solve((n, 1, 1), coef, b, "bicgstab_jacobi", RTOL, 7)
    else:
        col = np.arange(n) + np.where(even, 1, -1)
        x, its, rr, st = _lib.csr_solve(np.arange(n + 1), col, np.where(even, 1.0, -1.0), b, "bicgstab_jacobi", RTOL, 0.0, 7)
        assert st == 2 and its == 7 and rr == 1.0
        assert not x.any()


@pytest.mark.parametrize("method", ["bicgstab_jacobi", "cg_jacobi"])
@pytest.mark.parametrize("width", [1, 7, 8, 9, 21])
@pytest.mark.parametrize("n", [21, 3001, 8000, 16384, 20011, 33000])
def test_compressed_rows_shorter_and_longer_than_the_registers_hold(n, width, method):
    """Rows of 1 to `width` entries that reach over the whole matrix, symmetric for CG; the bound is the
    stopping test's, as above."""
    rng = np.random.default_rng(n + width)
    if method == "cg_jacobi":   # symmetric: pairs (i, n - 1 - i) and bands, each entry with its mirror image
        offs = np.unique(np.concatenate([[0], *[[-o, o] for o in rng.integers(1, n, (width - 1) // 2)]]).astype(int))
        rows = [np.unique(np.clip(i + offs, 0, n - 1)[(i + offs >= 0) & (i + offs < n)]) for i in range(n)]
        vals = [np.where(c == i, 2.0 * width, -1.0) for i, c in enumerate(rows)]
    else:
        rows = [np.unique(np.append(rng.integers(0, n, rng.integers(0, width)), i)) for i in range(n)]
        vals = [np.where(c == i, 2.0 * width, rng.uniform(-1.0, 1.0, c.size)) for i, c in enumerate(rows)]
    ptr = np.concatenate([[0], np.cumsum([c.size for c in rows])])
    col, val, b = np.concatenate(rows), np.concatenate(vals), rng.standard_normal(n)
    x, _, rr, st = _lib.csr_solve(ptr, col, val, b, method, RTOL)
    assert st == 0 and rr <= RTOL
    ax = np.add.reduceat(val * x[col], ptr[:-1])
    assert np.linalg.norm(b - ax) <= 1e-11 * np.linalg.norm(b)
