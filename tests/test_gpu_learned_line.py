"""The level pyramid of a very long, thin lattice: its twelve levels end far above the 64 cells at which
others stop, and the coarse levels do not fit the shared memory that a launch may take unasked."""
import numpy as np
import pytest

from caffe_old_b200 import cases as C, precond as P
from caffe_old_b200.solver import make_solver

pytestmark = pytest.mark.gpu


def test_a_line_of_thirteen_million_cells_runs_the_pyramid():
    n = (13_000_000, 1, 1)
    assert np.prod(P.pyramid_dims(n)[-1]) > 6144
    x = np.linspace(0.0, 1.0, n[0] + 1)
    nodes = np.zeros((2, 2, n[0] + 1, 3))
    nodes[..., 0] = x
    nodes[:, 1, :, 1] = nodes[1, :, :, 2] = 1e-3
    bc, ref = C.channel_bcs(1.0)
    spec = C.CaseSpec(kind="piso", bc=bc, ref_vec=ref, rho=1.0, mu=0.01, time_accurate=True, omega_u=1.0, omega_p=1.0, n_inner=1, n_pcorr=1,
                      convection="upwind", mom_method="bicgstab_jacobi", p_method="cg_jacobi", mom_rtol=1e-8, p_rtol=1e-8, maxit=4,
                      dt=1e-3, p_form="learned_mixed")
    d = make_solver(nodes, spec)
    P.set_mode(d, "levels")
    for ph in ("save_u0", "assemble_momentum", "solve_momentum", "momentum_post", "assemble_pcorr", "solve_pcorr"):
        d.phase(ph)
    assert np.isfinite(d.field("pCorr")).all()
