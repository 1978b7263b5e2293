"""The resident SOR launch (default sweeps of grids that fit the SMs' shared
memory) against the separate sweeps: same iterates, counts and norms, bit for
bit, at the edges of its blocks and groups."""
import numpy as np
import pytest

import hydrocode_astro1_b200 as hc

pytestmark = pytest.mark.gpu

# one cell per row pair, one-row and one-plane blocks, rows of partial vectors,
# an odd count of rows per block, the largest FP64 cube that fits, one that does not
SHAPES = [(3, 3, 3), (4, 3, 9), (3, 40, 5), (90, 4, 6), (20, 18, 22), (23, 31, 67), (17, 200, 14), (150, 151, 148),
          (158, 157, 160)]


def solve64(shape, depth, max_iter, tol, seed=1):
    rng = np.random.default_rng(seed)
    rho, phi = rng.random(shape) + 0.1, rng.standard_normal(shape)
    with hc.HydroSolver3D(shape, G=1.0, gravity_only=1, max_iter=max_iter, tol=tol, sor_depth=depth,
                          moment_order=hc.MOMENTS_TREE) as s:
        s.set_phi(phi)
        rc = s.gravity_solve(rho)
        d = s.diagnostics()
        return s.phi(), rc, d["last_iterations"], d["last_residual"]


@pytest.mark.parametrize("max_iter", [1, 2, 18, 45])
@pytest.mark.parametrize("shape", SHAPES)
def test_resident_fp64_capped(shape, max_iter):
    a, b = (solve64(shape, depth, max_iter, 1e-30) for depth in (0, -1))
    assert np.array_equal(a[0], b[0])
    assert a[1:] == b[1:]


# (1e3: the first iteration, which runs before the boundary values are set)
@pytest.mark.parametrize("tol", [1e3, 1e-2, 1e-3, 1e-5, 3e-7])
@pytest.mark.parametrize("shape", SHAPES[:7])
def test_resident_fp64_stops_at_the_same_iteration(shape, tol):
    a, b = (solve64(shape, depth, 20000, tol) for depth in (0, -1))
    assert np.array_equal(a[0], b[0])
    assert a[1:] == b[1:] and a[1] == hc.HC_OK


@pytest.mark.parametrize("shape", [(8, 7, 34), (20, 18, 22), (33, 70, 75), (61, 50, 99), (130, 20, 18)])
def test_resident_fp32_matches_sweeps(shape):
    # these rows are no whole vectors: sor_depth -2 runs the separate sweeps on them
    rng = np.random.default_rng(2)
    q = np.zeros((5,) + shape)
    q[0] = rng.random(shape) + 0.1
    q[4] = 1.0
    got = []
    for depth in (0, -2):
        with hc.HydroSolver3D(shape, G=1.0, precision=hc.FP32, max_iter=20000, tol=1e-6, sor_depth=depth,
                              moment_order=hc.MOMENTS_TREE) as s:
            s.set_state(q)
            rc = s.gravity_solve()
            d = s.diagnostics()
            got.append((s.phi(), rc, d["last_iterations"], d["last_residual"], d["outer_cycles"]))
    assert np.array_equal(got[0][0], got[1][0])
    assert got[0][1:] == got[1][1:]


def test_known_divisor_division_is_exact():
    # tiny, zero and huge right-hand sides leave the multiplying range of the
    # FP64 quotient; the result is the division's all the same
    shape = (12, 11, 14)
    rng = np.random.default_rng(4)
    out = []
    for depth in (0, 1):
        got = []
        for scale in (0.0, 1e-300, 1e-280, 1.0, 1e250, 1e290):
            with hc.HydroSolver3D(shape, G=1.0, gravity_only=1, max_iter=30, tol=1e-300, sor_depth=depth,
                                  moment_order=hc.MOMENTS_TREE, grav_bc=2) as s:
                s.set_phi(np.random.default_rng(5).standard_normal(shape) * scale)
                s.gravity_solve(np.abs(rng.standard_normal(shape)) * scale)
                got.append(s.phi())
        rng = np.random.default_rng(4)
        out.append(got)
    want = []
    for k, scale in enumerate((0.0, 1e-300, 1e-280, 1.0, 1e250, 1e290)):
        with hc.HydroSolver3D(shape, G=1.0, gravity_only=1, max_iter=30, tol=1e-300, sor_depth=-1,
                              moment_order=hc.MOMENTS_TREE, grav_bc=2) as s:
            s.set_phi(np.random.default_rng(5).standard_normal(shape) * scale)
            s.gravity_solve(np.abs(rng.standard_normal(shape)) * scale)
            want.append(s.phi())
    for got in out:
        for a, b in zip(got, want):
            assert np.array_equal(a, b)
