"""The learned p' solve with FGMRES on lattices whose cell count is not a multiple of four: the Krylov
basis planes are then further apart than the lattice's own plane stride.  Fields against the FP64
oracle, with the bounds of test_gpu_learned.py."""
import pytest

from oracle.oracle import OracleSolver
from caffe_old_b200 import precond as P
from caffe_old_b200.solver import make_solver

from helpers import demean, rel_l2, small_channel_sphere
from test_gpu_learned import FIELD_RTOL, P_RTOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(45, 15, 15), (45, 16, 15)])
@pytest.mark.parametrize("mode", ["levels", "network"])
def test_fgmres_on_odd_cell_counts(n, mode):
    nodes, spec = small_channel_sphere(n=n)
    o = OracleSolver(nodes, spec)
    d = make_solver(nodes, spec.replace(p_form="learned_mixed", p_rtol=P_RTOL, mom_rtol=1e-10))
    P.set_params(d, P.identity_params(1))
    P.set_mode(d, mode)
    P.set_options(d, "fgmres")
    for _ in range(2):
        o.solve()
        d.solve()
        st = d.last_stats
        assert st["status"] == 0 and st["p_res_max"] <= P_RTOL, st
    vol, mask = o.get("vol"), o.get("status") != 2
    assert rel_l2(d.field("u"), o.get("u")) < FIELD_RTOL
    assert rel_l2(demean(d.field("p"), vol, mask), demean(o.get("p"), vol, mask)) < FIELD_RTOL
