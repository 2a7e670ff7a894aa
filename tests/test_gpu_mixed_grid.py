"""The mixed form on the systems that run FP32 CG with reliable updates (symmetric, more than 32768 cells),
and what a handle holds for it."""
import numpy as np
import pytest

from oracle.oracle import OracleSolver
from caffe_old_b200.solver import make_solver

from helpers import demean, rel_l2, small_cavity3d, small_channel_sphere, small_skewed
from test_gpu_mixed import MIXED_FIELD_RTOL, P_RTOL

pytestmark = pytest.mark.gpu


def held(spec, nodes):
    """Bytes of device memory that a handle takes."""
    import torch
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    d = make_solver(nodes, spec)
    used = free - torch.cuda.mem_get_info()[0]
    d.close()
    return used


@pytest.mark.parametrize("maker,n,planes", [(small_cavity3d, (32, 32, 32), 0), (small_channel_sphere, (160, 60, 60), 0),
                                            (small_cavity3d, (96, 80, 80), 8)])
def test_fp32_planes_are_held_where_the_fp32_solve_runs(maker, n, planes):
    """Eight FP32 planes; the allocator hands out whole 2 MB blocks, so a handle may take one more for each."""
    nodes, spec = maker(n=n)
    held(spec, nodes)
    extra = held(spec.replace(p_form="mixed"), nodes) - held(spec, nodes)
    cells = int(np.prod(n))
    assert 4 * cells * planes <= extra <= 4 * cells * planes * 1.1 + planes * (2 << 20)


def test_sphere_without_ghost_rows_runs_the_fp32_solve():
    """A sphere outside the lattice leaves the system symmetric."""
    nodes, spec = small_channel_sphere(n=(48, 32, 28))
    spec = spec.replace(ib_center=(50.0, 0.5, 0.5), p_rtol=P_RTOL, mom_rtol=1e-10)
    d, e = make_solver(nodes, spec.replace(p_form="mixed")), make_solver(nodes, spec)
    for _ in range(2):
        d.solve()
        e.solve()
        assert d.last_stats["status"] == e.last_stats["status"] == 0 and d.last_stats["n_ghost"] == 0
        assert d.last_stats["p_res_max"] <= P_RTOL and d.last_stats["fallbacks"] == 0
    assert rel_l2(d.field("u"), e.field("u")) < MIXED_FIELD_RTOL


@pytest.mark.parametrize("maker,n", [(small_cavity3d, (36, 32, 30)), (small_cavity3d, (35, 33, 31)), (small_skewed, (36, 32, 30)),
                                     (small_skewed, (35, 33, 31)), (small_channel_sphere, (92, 24, 22))])
def test_mixed_precision_fields_match_fp64_oracle_above_one_cluster(maker, n):
    """Rows of whole and of odd length (four cells per thread and one), and a sphere, whose mixed form is the
    FP64 BiCGStab; bounds of test_gpu_mixed.py."""
    nodes, spec = maker(n=n)
    assert np.prod(n) > 32768
    o = OracleSolver(nodes, spec.replace(mom_rtol=1e-11, p_rtol=1e-11))
    d = make_solver(nodes, spec.replace(p_form="mixed", p_rtol=P_RTOL, mom_rtol=1e-10))
    for _ in range(2):
        o.solve()
        d.solve()
        st = d.last_stats
        assert st["status"] == 0 and st["fallbacks"] == 0, st
        assert st["p_res_max"] <= P_RTOL, st
    vol, mask = o.get("vol"), o.get("status") != 2
    assert rel_l2(d.field("u"), o.get("u")) < MIXED_FIELD_RTOL
    assert rel_l2(demean(d.field("p"), vol, mask), demean(o.get("p"), vol, mask)) < MIXED_FIELD_RTOL
    for nm in ("massFlowI", "massFlowJ", "massFlowK"):
        assert rel_l2(d.field(nm), o.get(nm)) < MIXED_FIELD_RTOL, nm
