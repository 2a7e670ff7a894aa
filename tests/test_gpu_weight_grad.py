"""The grouped weight gradient: one set of blocks works through the chunks of every lattice of a layer
and leaves one partial each.

* lattices at the edges of its split (one chunk, fewer chunks than a block's least share, more chunks
  than blocks) against the FP64 restatement, within the 2e-2 of the other network tests (bf16 rounding);
* one training step of the odd network term (net(x) - net(-x)) / 2, whose last-layer bias cancels: its
  gradient is round-off of an FP64 sum, far below the optimiser's epsilon of 1e-8, so the bias stays
  within 1e-3 of a step of where it was."""
import ctypes

import numpy as np
import pytest

from caffe_old_b200 import _lib, precond as P
from caffe_old_b200.solver import make_solver

import cnn_reference as R
from helpers import small_channel_sphere

pytestmark = pytest.mark.gpu
TOL = 2e-2


@pytest.mark.parametrize("shape", [(1, 1, 1), (16, 1, 1), (17, 3, 1), (5, 16, 3), (30, 45, 44)])
def test_gradient_at_the_edges_of_the_split(shape):
    n = int(np.prod(shape))
    rng = np.random.default_rng(9)
    params = R.random_params(6)
    x2 = rng.standard_normal((n, 2)).astype(np.float32)
    dy = rng.standard_normal(n).astype(np.float32)
    y = np.zeros(n, dtype=np.float32)
    g = np.zeros(4 * R.LAYER, dtype=np.float32)
    vp = ctypes.c_void_p
    rc = _lib.lib().caffe_precond_net_grad(*shape, params.ctypes.data_as(vp), x2.ctypes.data_as(vp), dy.ctypes.data_as(vp),
                                           y.ctypes.data_as(vp), g.ctypes.data_as(vp))
    assert rc == 0, _lib.last_error()
    _, gr = R.grad(params.astype(np.float64), x2.astype(np.float64), dy.astype(np.float64), shape)
    for l in range(4):
        blk = slice(l * R.LAYER, (l + 1) * R.LAYER)
        assert np.linalg.norm(g[blk] - gr[blk]) <= TOL * max(np.linalg.norm(gr[blk]), 1e-30), l


def test_cancelling_bias_stays_put_in_training():
    nodes, spec = small_channel_sphere(n=(48, 16, 16))
    s = make_solver(nodes, spec.replace(p_form="fp64"))
    s.solve()
    P.add_random_pairs(s, 4, seed=5)
    start = P.load_default()
    lr = 1e-3
    trained, _ = P.train(s, start, steps=1, batch=4, lr=lr, seed=1)
    last_bias = P.weight_view(trained, 3)[1][0] - P.weight_view(start, 3)[1][0]
    moved = np.abs(trained - start)
    assert moved.max() > 0.9 * lr
    assert abs(last_bias) <= 1e-3 * lr
