"""Which relaxation a default solve takes: grids that are mostly block edge or
mostly halo keep the separate sweeps (the resident launch and the streaming
passes measured up to four times slower there), the others do not; the iterates,
counts and norms are the same bits on every route."""
import numpy as np
import pytest

import hydrocode_astro1_b200 as hc

pytestmark = pytest.mark.gpu

RESIDENT, PASSES, SWEEPS = "resident", "passes", "sweeps"
ROUTES = [
    (hc.FP64, (4, 15, 4132), SWEEPS), (hc.FP64, (3, 3, 4000), SWEEPS), (hc.FP64, (20, 20, 1000), SWEEPS),
    (hc.FP64, (64, 64, 600), SWEEPS), (hc.FP64, (30, 60, 501), SWEEPS), (hc.FP64, (118, 3, 1059), RESIDENT),
    (hc.FP64, (3, 3, 300), RESIDENT), (hc.FP64, (20, 18, 22), RESIDENT), (hc.FP64, (128, 128, 128), RESIDENT),
    (hc.FP64, (400, 400, 6), RESIDENT), (hc.FP64, (160, 160, 160), SWEEPS),
    (hc.FP32, (23, 10, 5511), SWEEPS), (hc.FP32, (4, 103, 3901), SWEEPS), (hc.FP32, (64, 64, 600), PASSES),
    (hc.FP32, (12, 679, 436), RESIDENT), (hc.FP32, (128, 128, 128), RESIDENT), (hc.FP32, (192, 192, 192), RESIDENT),
    (hc.FP32, (6, 1132, 2048), SWEEPS), (hc.FP32, (2119, 9, 512), SWEEPS), (hc.FP32, (1024, 8, 2048), SWEEPS),
    (hc.FP32, (24, 946, 512), SWEEPS), (hc.FP32, (24, 5016, 128), PASSES), (hc.FP32, (256, 256, 256), PASSES),
    (hc.FP32, (250, 250, 250), SWEEPS),     # rows of an odd number of vectors
]


@pytest.mark.parametrize("precision,shape,route", ROUTES)
def test_route_and_bits(precision, shape, route):
    rng = np.random.default_rng(4)
    q = np.zeros((5,) + shape)
    q[0], q[4] = rng.random(shape) + 0.1, 1.0
    its, got = 24, []
    # FP32: -3 runs separate sweeps, staged by TMA where the rows allow it
    for depth in (0, -1 if precision == hc.FP64 else -3):
        with hc.HydroSolver3D(shape, G=1.0, precision=precision, max_iter=its, tol=1e-30, sor_depth=depth,
                              moment_order=hc.MOMENTS_TREE) as s:
            s.set_state(q)
            s.timing(reset=True)
            s.gravity_solve()
            launches, d = s.timing()["sor_launches"], s.diagnostics()
            got.append((s.phi(), d["last_iterations"], d["last_residual"]))
            if depth == 0:
                assert d["last_iterations"] == its
                assert route == (RESIDENT if launches < its / 4 else PASSES if launches <= its / 2 + 2 else SWEEPS)
    assert np.array_equal(got[0][0], got[1][0])
    assert got[0][1:] == got[1][1:]
