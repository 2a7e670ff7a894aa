"""Systems above 32768 cells that the scaled CG hands to the general one: a diagonal of mixed signs, a matrix
that is not symmetric, an entry that points beyond the lattice's end.  The entry point without
allocation has no planes for the scaled form, so its CG is the general one always: same bits, or the scaled
form ran.  Rows of whole and of odd length (two cells per thread and one)."""
import numpy as np
import pytest

from caffe_old_b200 import _lib

from test_zz_no_alloc import seven_point_residual, seven_point_system, solve_with

pytestmark = pytest.mark.gpu

SHAPES = [(40, 33, 32), (41, 33, 32)]


def both(shape, coef, b):
    L = _lib.lib()
    scaled = solve_with(L.caffe_ksp7_solve_device, shape, coef, b, "cg_jacobi")
    general = solve_with(L.caffe_ksp7_solve_device_noalloc, shape, coef, b, "cg_jacobi")
    return scaled, general


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kind", ["signs", "west", "south", "bottom", "beyond"])
def test_the_general_form_takes_what_the_scaled_one_cannot(shape, kind):
    coef, b = seven_point_system(shape, 4, True)
    coef = coef.copy()
    if kind == "signs":
        coef[1:] = 0.0
        coef[0] = np.where(np.arange(coef.shape[1]) % 3 == 0, 1.0, -1.0) * np.abs(coef[0])
    elif kind == "beyond":
        coef[5, -1] = 1.0   # the top entry of the last cell: multiplied by the zero halo
    else:
        coef[{"west": 2, "south": 4, "bottom": 6}[kind], -2] *= 1.0 + 1e-9
    (rc, x, _, rr), (rg, xg, _, _) = both(shape, coef, b)
    assert rc == 0 and rg == 0 and rr <= 1e-12
    coef[5, -1] = 0.0
    assert seven_point_residual(shape, coef, x, b) <= 1e-11
    assert np.array_equal(x, xg)


@pytest.mark.parametrize("sign", [-1.0, 1.0])
@pytest.mark.parametrize("shape", SHAPES)
def test_the_scaled_form_takes_the_rest(shape, sign):
    coef, b = seven_point_system(shape, 4, True)
    coef = sign * coef
    (rc, x, _, rr), (_, xg, _, _) = both(shape, coef, b)
    assert rc == 0 and rr <= 1e-12
    assert seven_point_residual(shape, coef, x, b) <= 1e-11
    assert not np.array_equal(x, xg) and np.linalg.norm(x - xg) <= 1e-9 * np.linalg.norm(xg)


@pytest.mark.parametrize("shape", SHAPES)
def test_bicgstab_without_allocation_on_the_grid(shape):
    """The same kernel on the other entry's workspace: same bits."""
    coef, b = seven_point_system(shape, 6, False)
    L = _lib.lib()
    rc, x, its, rr = solve_with(L.caffe_ksp7_solve_device, shape, coef, b, "bicgstab_jacobi")
    rg, xg, itg, _ = solve_with(L.caffe_ksp7_solve_device_noalloc, shape, coef, b, "bicgstab_jacobi")
    assert rc == 0 and rg == 0 and rr <= 1e-12 and its == itg
    assert seven_point_residual(shape, coef, x, b) <= 1e-11
    assert np.array_equal(x, xg)
