"""When the Krylov kernels restart from the true residual, and when they must not: in one cluster (up
to 32768 rows) and on the grid (above)."""
import numpy as np
import pytest

from caffe_old_b200 import _lib, precond as P
from caffe_old_b200 import cases as C
from caffe_old_b200.solver import make_solver

from helpers import small_cavity2d, small_cavity3d
from test_zz_no_alloc import seven_point_residual, seven_point_system

pytestmark = pytest.mark.gpu


def pressure_solve(d, b):
    """p' of the handle's assembled system for the right-hand side b, and the solve's statistics."""
    d.set_field("pcB", b)
    d.phase("solve_pcorr")
    return d.field("pCorr"), d.stats()


@pytest.mark.parametrize("n", [(36, 32, 32), (34, 33, 31), (33, 32, 32)])
def test_restarts_of_a_singular_system_repeat_bit_for_bit(n):
    """All-Neumann cavity, CG: a relative tolerance of 1e-17 lies below round-off, so the recursive residual
    passes it again and again and the solve restarts, projected, until maxit.  Every row parity: the
    sweeps take two cells per thread where rows are even, the restart one.  Bound of the residual: round-off
    at a condition number of about 1e3 (1e-13) times the 1e3 by which it may rise before a restart, and ten."""
    nodes, spec = small_cavity3d(n=n)
    d = make_solver(nodes, spec.replace(p_rtol=1e-17, maxit=3000))
    for ph in ("save_u0", "assemble_momentum", "solve_momentum", "momentum_post", "assemble_pcorr"):
        d.phase(ph)
    b = np.random.default_rng(1).standard_normal(d.ncells)
    first, st = pressure_solve(d, b)
    assert st["p_iters_last"] == 3000 and st["p_res_max"] <= 1e-9
    for _ in range(5):
        again, st = pressure_solve(d, b)
        assert np.array_equal(again, first)


@pytest.mark.parametrize("shape", [(20, 20, 20), (64, 64, 1), (31, 30, 29), (36, 32, 32), (33, 33, 33)])
def test_cg_converges_on_a_nearly_singular_matrix(shape):
    """Row sums of 1e-9: (r, r) rises far above its start before it falls, which is no reason to restart.
    A solve takes a few hundred iterations; the residual is the stopping test's, evaluated on the host."""
    coef, b = seven_point_system(shape, 21, True)
    coef[0] = -coef[1:].sum(axis=0) - 1e-9
    x, its, rr, st = _lib.ksp7_solve(shape, coef, b, "cg_jacobi", 1e-8, 2000)
    assert st == 0 and rr <= 1e-8
    assert seven_point_residual(shape, coef, x, b) <= 1.1e-8


def convective_system(shape, seed, pe):
    """Upwind convection in a rotating flow of cell Peclet number up to pe / 2, with a little reaction."""
    nI, nJ, nK = shape
    N = nI * nJ * nK
    idx = np.arange(N)
    i, j, k = idx % nI, (idx // nI) % nJ, idx // (nI * nJ)
    u, v = pe * (j / nJ - 0.5), -pe * (i / nI - 0.5)     # through a cell's east and west, north and south faces
    coef = np.zeros((7, N))
    for q, (inside, into) in enumerate(((i < nI - 1, -u), (i > 0, u), (j < nJ - 1, -v), (j > 0, v), (k < nK - 1, 0 * u), (k > 0, 0 * u))):
        coef[q + 1][inside] = (1.0 + np.maximum(into, 0.0))[inside]
    coef[0] = -coef[1:].sum(axis=0) - 1e-3
    return coef, np.random.default_rng(seed).standard_normal(N)


@pytest.mark.parametrize("shape,peclets,most", [((64, 64, 1), (10.0, 30.0, 100.0, 300.0), 187_000), ((40, 36, 30), (10.0, 30.0), 112_000)])
def test_bicgstab_restarts_on_an_almost_vanishing_rho(shape, peclets, most):
    """Convective systems on which (rp, r) sinks to round-off.  How long one of them takes is chance; together,
    with (rp, r) summed over the cells in every iteration, they take 124,500 and 75,000 iterations, and
    the bound is half as many again (over 290,000 without the restarts, and some end at maxit).  The
    residual is the stopping test's, evaluated on the host."""
    total = 0
    for pe in peclets:
        for seed in range(12):
            coef, b = convective_system(shape, seed, pe)
            x, its, rr, st = _lib.ksp7_solve(shape, coef, b, "bicgstab_jacobi", 1e-9, 20000)
            assert st == 0 and rr <= 1e-9
            assert seven_point_residual(shape, coef, x, b) <= 1.1e-9
            total += its
    assert total <= most


def test_fp64_solve_behind_a_failed_learned_one_converges_on_a_large_lattice():
    """Network parameters that are not numbers: every learned solve of the step fails at once, and the FP64
    BiCGStab behind it solves the systems of a 6.3M-cell sphere, from rest."""
    nodes, spec, _ = C.config5_sphere((240, 160, 164), p_form="learned_mixed")
    d = make_solver(nodes, spec)
    P.set_params(d, np.full_like(P.load_default(), np.nan))
    P.set_mode(d, "network")
    d.solve()
    st = d.last_stats
    assert st["fallbacks"] == st["p_solves"] > 0
    assert st["p_res_max"] <= spec.p_rtol


@pytest.mark.parametrize("block,rhs", [([[-1, -1, 0], [2, 1, 0], [0, 2, -1]], [0, -1, -1]), ([[-1, -2, 0], [0, 1, -1], [0, 2, -1]], [-1, 1, 0])])
@pytest.mark.parametrize("blocks", [3, 10000, 16384])
def test_bicgstab_restarts_where_rho_is_exactly_zero(block, rhs, blocks):
    """Blocks of three rows, all values small whole numbers or halves: after the first iteration x is finite, r is
    not zero and (rp, r) is exactly zero in any order of summation; going on, the second beta is 0 / 0 and
    the next direction not a number.  The solve restarts from the true residual with the x it has and takes a
    few iterations more (condition numbers below 100)."""
    block, rhs = np.array(block, dtype=float), np.array(rhs, dtype=float)
    coef = np.zeros((7, 3 * blocks))
    coef[0] = np.tile(np.diag(block), blocks)
    coef[1] = np.tile([block[0, 1], block[1, 2], 0.0], blocks)
    coef[2] = np.tile([0.0, block[1, 0], block[2, 1]], blocks)
    x, _, rr, st = _lib.ksp7_solve((3 * blocks, 1, 1), coef, np.tile(rhs, blocks), "bicgstab_jacobi", 1e-12, 50)
    assert st == 0 and rr <= 1e-12
    assert np.linalg.norm(x.reshape(blocks, 3) - np.linalg.solve(block, rhs)) <= 1e-10 * np.linalg.norm(x)


@pytest.mark.parametrize("n,m", [(24, 20), (64, 64), (150, 120), (190, 180)])
def test_bicgstab_of_a_singular_system_ignores_the_mean_of_its_right_hand_side(n, m):
    """All-Neumann cavity; whole numbers of mean zero, and the same shifted by 2^46 (exact in FP64): the mean is
    projected out before the solve starts, so both take the same iterations but for round-off."""
    nodes, spec = small_cavity2d(n, m)
    d = make_solver(nodes, spec.replace(p_rtol=1e-8, maxit=20000))
    for ph in ("save_u0", "assemble_momentum", "solve_momentum", "momentum_post", "assemble_pcorr"):
        d.phase(ph)
    b = np.random.default_rng(2).integers(-8, 9, d.ncells // 2).astype(float)
    b = np.concatenate([b, -b])
    x0, st0 = pressure_solve(d, b)
    x1, st1 = pressure_solve(d, b + 2.0**46)
    assert st0["p_res_max"] <= 1e-8 and st1["p_res_max"] <= 1e-8
    assert st1["p_iters_last"] <= 1.2 * st0["p_iters_last"] + 5
    assert np.linalg.norm(x1 - x0) <= 1e-4 * np.linalg.norm(x0)


@pytest.mark.parametrize("method", ["bicgstab_jacobi", "cg_jacobi"])
@pytest.mark.parametrize("shape", [(20, 20, 20), (36, 32, 32)])
def test_right_hand_sides_of_any_size_take_the_same_iterations(shape, method):
    """Scaled by a power of two every number of a solve scales exactly, up to where the square of a squared norm
    leaves the range: the restart rules must not see the difference."""
    coef, b = seven_point_system(shape, 8, method == "cg_jacobi")
    x, its, _, st = _lib.ksp7_solve(shape, coef, b, method, 1e-10, 5000)
    assert st == 0
    for e in (-300, 300):
        xs, itss, _, st = _lib.ksp7_solve(shape, coef, b * 2.0**e, method, 1e-10, 5000)
        assert st == 0 and itss == its
        assert np.array_equal(xs, x * 2.0**e)


@pytest.mark.parametrize("shape", [(5, 4, 3), (10, 10, 10), (20, 20, 20), (32, 32, 32), (36, 32, 32)])
@pytest.mark.parametrize("kind", ["zero entry", "one sign turned", "a strip turned", "random signs"])
def test_cg_with_a_diagonal_that_is_not_of_one_sign(shape, kind):
    """(r, D^-1 r) changes sign there and beta with it.  Up to 180 iterations; ten times that are allowed."""
    coef, b = seven_point_system(shape, 8, True)
    N = b.size
    if kind == "zero entry":
        coef[0, 7] = 0.0
    elif kind == "one sign turned":
        coef[0, N // 2] *= -1.0
    elif kind == "a strip turned":
        coef[0, :N // 8] *= -1.0
    else:
        coef[1:] *= 0.3
        coef[0] *= np.where(np.random.default_rng(8).random(N) < 0.3, -1.0, 1.0)
    x, _, rr, st = _lib.ksp7_solve(shape, coef, b, "cg_jacobi", 1e-10, 1800)
    assert st == 0 and rr <= 1e-10
    assert seven_point_residual(shape, coef, x, b) <= 1.1e-10
