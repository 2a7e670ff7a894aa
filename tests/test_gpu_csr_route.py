"""Which compressed-row systems one thread-block cluster solves: a solve there is one launch, on the whole
grid two (1/d, then the solver).  Rows beyond what the cluster's threads hold in registers, and more than two rows
per thread, are faster on the grid."""
import numpy as np
import pytest

from caffe_old_b200 import _lib
from caffe_old_b200.solver import Coupled

from test_gpu_coupled import CASES

pytestmark = pytest.mark.gpu


def banded(n, entries):
    """Rows of `entries` entries around the diagonal (cyclic), diagonally dominant."""
    off = np.arange(entries) - entries // 2
    col = (np.arange(n)[:, None] + off) % n
    val = np.where(off == 0, 2.0 * entries, -1.0 - 0.1 * (off > 0)) * np.ones((n, 1))
    return np.arange(n + 1) * entries, col.ravel(), val.ravel()


def launches(call):
    before = _lib.lib().caffe_launch_count()
    call()
    return _lib.lib().caffe_launch_count() - before


@pytest.mark.parametrize("method", ["bicgstab_jacobi", "cg_jacobi"])
@pytest.mark.parametrize("n,entries,cluster", [(100, 5, True), (8192, 14, True), (8192, 15, False), (8193, 9, True), (16384, 9, True),
                                               (16384, 10, False), (16385, 1, False), (16385, 5, False), (32768, 14, False)])
def test_long_rows_and_many_rows_leave_the_cluster(n, entries, cluster, method):
    ptr, col, val = banded(n, entries)
    if method == "cg_jacobi":
        if entries % 2 == 0:
            pytest.skip("a band with one entry more on one side is not symmetric")
        val = np.where(val < 0, -1.0, val)
    b = np.random.default_rng(entries).standard_normal(n)

    def solve():
        x, _, rr, st = _lib.csr_solve(ptr, col, val, b, method, 1e-12)
        assert st == 0 and rr <= 1e-12
        assert np.linalg.norm(b - np.add.reduceat(val * x[col], ptr[:-1])) <= 1e-11 * np.linalg.norm(b)

    assert launches(solve) == (2 if cluster else 3)   # with the search for the diagonals


def test_the_coupled_block_rows_run_on_the_grid():
    """Continuity rows of 20 and 28 entries."""
    nodes, spec = CASES["skewed3d"]()
    d = Coupled(nodes, spec)
    for ph in ("save_u0", "assemble"):
        d.phase(ph)
    assert launches(lambda: d.phase("solve")) == 2
