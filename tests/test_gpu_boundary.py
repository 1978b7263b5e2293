"""The face cells of a step -- source, periodic copies and conditions resolved
in one launch -- against the oracle, which applies them one after the other:
every kind on every face, grids down to three cells, and the tile origins of
the interior update (a last tile of one column or row)."""
import itertools

import numpy as np
import pytest

import hydrocode_astro1_b200 as hc
import ics
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu

MIXED = [(0, 0, 1, 2, 2, 1), (2, 1, 0, 0, 1, 1), (1, 2, 2, 1, 0, 0), (0, 0, 0, 0, 1, 2), (1, 1, 0, 0, 0, 0),
         (0, 1, 2, 0, 1, 0), (0, 2, 0, 1, 0, 2)]


@pytest.mark.parametrize("shape", [(3, 3, 3), (5, 4, 3), (9, 10, 34), (6, 18, 33)])
@pytest.mark.parametrize("bc", [(t,) * 6 for t in (0, 1, 2)] + MIXED)
@pytest.mark.parametrize("G", [0.0, 1.0])
def test_faces_bitwise(shape, bc, G):
    q0 = ics.smooth_random(shape, seed=5)
    kw = dict(G=G, cfl=0.3, bc=bc, tol=1e-3, max_iter=50)
    o = OracleSim(*shape, **kw)
    o.set_state(q0)
    d_o, _, _ = o.step(4)
    with hc.HydroSolver3D(shape, **kw) as s:
        s.set_state(q0)
        d = s.step(4)
        assert np.array_equal(d, d_o)
        assert np.array_equal(s.state(), o.state())


@pytest.mark.parametrize("shape", list(itertools.product((7,), (9, 10, 11, 17), (33, 34, 35, 65))))
def test_tile_origins_bitwise(shape):
    q0 = ics.smooth_random(shape, seed=6)
    o = OracleSim(*shape, cfl=0.3)
    o.set_state(q0)
    d_o, _, _ = o.step(3)
    with hc.HydroSolver3D(shape, cfl=0.3) as s:
        s.set_state(q0)
        assert np.array_equal(s.step(3), d_o)
        assert np.array_equal(s.state(), o.state())
