"""When the Krylov kernels restart from the true residual, and when they must not: in one cluster (up
to 32768 rows) and on the grid (above)."""
import numpy as np
import pytest

from caffe_old_b200 import _lib
from caffe_old_b200.solver import make_solver

from helpers import small_cavity3d
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
