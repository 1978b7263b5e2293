"""The streaming SOR passes (default FP32 correction sweeps of grids that do
not fit the SMs' shared memory) against the separate sweeps: same iterates,
counts and norms, bit for bit, on rows that need one and several tiles and odd
counts of iterations."""
import numpy as np
import pytest

import hydrocode_astro1_b200 as hc

pytestmark = pytest.mark.gpu

# sor_depth -3 runs the separate sweeps (staged by TMA up to 256 cells per
# colour and row)
@pytest.mark.parametrize("shape", [(1300, 60, 128), (50, 70, 2400), (60, 1700, 80), (210, 205, 208), (230, 180, 231)])
@pytest.mark.parametrize("tol,max_iter", [(1e-30, 1), (1e-30, 20), (1e-30, 35), (3e-4, 2000), (2e-4, 2000)])
def test_stream_fp32_matches_sweeps(shape, tol, max_iter):
    rng = np.random.default_rng(3)
    q = np.zeros((5,) + shape)
    q[0] = rng.random(shape) + 0.1
    q[4] = 1.0
    got = []
    for depth in (0, -3):
        with hc.HydroSolver3D(shape, G=1.0, precision=hc.FP32, max_iter=max_iter, tol=tol, sor_depth=depth,
                              moment_order=hc.MOMENTS_TREE) as s:
            s.set_state(q)
            rc = s.gravity_solve()
            d = s.diagnostics()
            got.append((s.phi(), rc, d["last_iterations"], d["last_residual"], d["outer_cycles"]))
    assert np.array_equal(got[0][0], got[1][0])
    assert got[0][1:] == got[1][1:]
