"""Restarts of the pressure solve's Krylov kernels from the true residual, on systems above the 32768
cells that one cluster holds."""
import numpy as np
import pytest

from caffe_old_b200.solver import make_solver

from helpers import small_cavity3d

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
