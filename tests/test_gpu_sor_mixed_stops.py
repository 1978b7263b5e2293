"""Mixed-precision solves to convergence on rows of whole vectors, of an even and
an odd number of cells: the resident launch (stops inside its groups) and, with
the learned start leaving its prediction in the second correction buffer, the
streaming passes, against the TMA-staged separate sweeps (sor_depth -3), bit for
bit."""
import os

import numpy as np
import pytest

import hydrocode_astro1_b200 as hc

pytestmark = pytest.mark.gpu

WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(hc.__file__)), "data", "unet_stellar_explosion_256.bin")


@pytest.mark.parametrize("shape", [(64, 60, 64), (96, 96, 96), (70, 70, 71), (9, 150, 87), (150, 7, 32), (130, 128, 192)])
@pytest.mark.parametrize("tol", [1e-4, 1e-6])
def test_resident_stops(shape, tol):
    rng = np.random.default_rng(6)
    q = np.zeros((5,) + shape)
    q[0], q[4] = rng.random(shape) + 0.1, 1.0
    phi = 0.1 * rng.standard_normal(shape)
    got = []
    for depth in (0, -3):
        with hc.HydroSolver3D(shape, G=1.0, precision=hc.FP32, max_iter=20000, tol=tol, sor_depth=depth,
                              moment_order=hc.MOMENTS_TREE) as s:
            s.set_state(q)
            s.set_phi(phi)
            runs = []
            for scale in (1.0, 1.001):      # a long solve and a short one
                s.set_state(q * scale)
                rc = s.gravity_solve()
                d = s.diagnostics()
                runs.append((s.phi(), (rc, d["last_iterations"], d["last_residual"], d["outer_cycles"])))
            launches = s.timing()["sor_launches"]
            assert depth != 0 or launches < sum(r[1][1] for r in runs) / 2
            got.append(runs)
    for a, b in zip(*got):
        assert np.array_equal(a[0], b[0]) and a[1] == b[1]


def test_learned_start_then_passes():
    shape = (224, 224, 192)      # more cells than the resident launch holds
    x = np.meshgrid(*[(np.arange(n) + 0.5) * 1.5 / n - 0.75 for n in shape], indexing="ij", sparse=True)
    r2 = sum(v * v for v in x)
    q = np.zeros((5,) + shape)
    q[0] = np.maximum(1e-6, 1 - r2 / 0.16) * np.exp(0.01 * np.random.default_rng(7).standard_normal(shape))
    q[4] = 1.5 * q[0] ** (5 / 3) + 200.0 * (r2 < 0.002)
    got = []
    for depth in (0, -3):
        with hc.HydroSolver3D(shape, lo=(-0.75,) * 3, hi=(0.75,) * 3, G=1.0, lmax=4, precision=hc.FP32, tol=1e-6,
                              max_iter=20000, sor_depth=depth, warm_start=hc.WARM_UNET,
                              moment_order=hc.MOMENTS_TREE) as s:
            s.unet_load_file(WEIGHTS)
            s.set_state(q)
            dts = s.step(4)
            d = s.diagnostics()
            got.append((s.state(), s.phi(), dts, d["total_iterations"], d["unet_accepted"], d["unet_fallbacks"]))
    assert got[0][4] + got[0][5] > 0      # it predicted
    for a, b in zip(*got):
        assert np.array_equal(a, b)
