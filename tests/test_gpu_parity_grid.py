"""Whole steps against the CPU oracle on lattices above the 32768 cells that one cluster holds: the grid's CG
(two cells per thread and one), its BiCGStab with and without ghost rows and with a projected right-hand
side, and the three-sided momentum solve.  Tolerances of test_gpu_parity.py."""
import numpy as np
import pytest

from oracle.oracle import OracleSolver
from caffe_old_b200.solver import make_solver

from helpers import (FIELD_RTOL, demean, rel_l2, small_cavity3d, small_channel_sphere, small_outlet_top, small_simple_transient,
                     small_skewed)

pytestmark = pytest.mark.gpu


def cavity_bicgstab(n):
    return small_cavity3d(n, cg=False)


@pytest.mark.parametrize("maker,n,steps", [(small_cavity3d, (36, 32, 30), 3), (small_cavity3d, (35, 33, 31), 3), (cavity_bicgstab, (36, 32, 30), 2),
                                           (small_skewed, (36, 32, 30), 2), (small_skewed, (35, 33, 31), 2),
                                           (small_channel_sphere, (92, 24, 22), 2), (small_simple_transient, (34, 33, 31), 2),
                                           (small_outlet_top, (26, 25, 52), 3)])
def test_steps_match_oracle_above_one_cluster(maker, n, steps):
    nodes, spec = maker(n=n)
    assert np.prod(n) > 32768
    # a cavity's p' system solved by BiCGStab on the device: the oracle takes its CG for it (at 1e-13 its own
    # BiCGStab ends in NaN on this singular system)
    o = OracleSolver(nodes, spec.replace(p_method="cg_jacobi") if maker is cavity_bicgstab else spec)
    d = make_solver(nodes, spec)
    for _ in range(steps):
        o.solve()
        d.solve()
        assert d.last_stats["status"] == 0, d.last_stats
    vol = o.get("vol")
    mask = o.get("status") != 2
    assert rel_l2(d.field("u"), o.get("u")) < FIELD_RTOL
    assert rel_l2(demean(d.field("p"), vol, mask), demean(o.get("p"), vol, mask)) < FIELD_RTOL
    for nm in ("massFlowI", "massFlowJ", "massFlowK"):
        assert rel_l2(d.field(nm), o.get(nm)) < FIELD_RTOL, nm
