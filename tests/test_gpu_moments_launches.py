"""The kernels that the moments in the reference's order count as launched: one
for a grid that is added cell by cell, the records' sixteen above, seven or one
per pass of a slab."""
import ctypes as C

import numpy as np
import pytest

import hydrocode_astro1_b200 as hc

pytestmark = pytest.mark.gpu


def launches(shape, order):
    with hc.HydroSolver3D(shape, G=1.0, gravity_only=1, max_iter=1, tol=1e-30, moment_order=order) as s:
        rho = np.ones(shape)
        s.gravity_solve(rho)
        s.timing(reset=True)
        s.gravity_solve(rho)
        return s.timing()["launches"]


# tree moments: four kernels on every grid
@pytest.mark.parametrize("shape,count", [((20, 18, 22), 1), ((27, 27, 27), 1), ((28, 28, 28), 16), ((64, 64, 64), 16)])
def test_launches_counted(shape, count):
    assert launches(shape, hc.MOMENTS_SEQUENTIAL) - launches(shape, hc.MOMENTS_TREE) == count - 4


@pytest.mark.parametrize("shape,count", [((12, 18, 22), 1), ((40, 30, 32), 7)])
def test_slab_launches_counted(shape, count):
    L = hc.lib()
    with hc.HydroSolver3D(shape, G=1.0) as s:
        q = np.zeros((5,) + shape)
        q[0] = q[4] = 1.0
        s.set_state(q)
        assert L.hc_set_slab(s.h, shape[0], 0) == hc.HC_OK
        sums = (C.c_double * 9)()
        s.timing(reset=True)
        assert L.hc_slab_moments(s.h, 0, sums) == hc.HC_OK
        assert s.timing()["launches"] == count
