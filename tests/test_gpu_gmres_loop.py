"""Solves of more steps than one launch of the device loop takes (512), with a restart at the end of a
launch: the loop that goes on must be where the host-driven one (h2b_solve_gmres_noalloc) is.  Both
restart every kmax - 1 steps, a divisor of 512 here, so that the 512th step restarts.  Sums in another
order move the step at which an estimate passes 1e-8 by a few of several hundred: 2 %."""
import numpy as np
import pytest

from h2lib_b200 import bem3d as hb
from test_zz_no_alloc import relerr, solve_noalloc

pytestmark = pytest.mark.gpu
L, C = hb.BASIS_LINEAR_BEM3D, hb.BASIS_CONSTANT_BEM3D


@pytest.mark.parametrize("basis,kmax", [(C, 3), (L, 5)])
def test_restart_at_the_end_of_a_launch(basis, kmax):
    gr = hb.new_ellipsoid_surface3d(6, (1.0, 0.7, 1.4))
    op = hb.new_slp_laplace_bem3d(gr, 2, 4, basis, basis)
    V = hb.H2Matrix(op, hb.build_tree(gr, basis, basis, 16, 1.4), 3).assemble()
    b = np.random.default_rng(1).standard_normal(V.rows)
    ref, y = solve_noalloc([V], [1.0], b, 1e-8, 4000, kmax)
    x = np.zeros(V.rows)
    it = hb.solve_gmres([V], [1.0], b, x, 1e-8, 4000, kmax)
    assert 512 < it and abs(it - ref) <= 0.02 * ref
    assert hb.residual_norm([V], [1.0], b, x) <= 1.001e-8
    assert relerr(x, y) < 1e-5
