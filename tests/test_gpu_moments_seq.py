"""Moments in the reference's summation order: the records of runs of cells
against the oracle's cell-by-cell sums, bit for bit -- sums that keep their
sign, that oscillate about zero, that tie at every cell, and inputs the
records do not cover."""
import numpy as np
import pytest

import hydrocode_astro1_b200 as hc
from oracle.oracle import OracleSim

pytestmark = pytest.mark.gpu

UNIT, CENTRED = ((0, 0, 0), (1, 1, 1)), ((-1, -1, -1), (1, 1, 1))


def density(kind, shape):
    rng = np.random.default_rng(7)
    if kind == "random":
        return rng.random(shape) + 1e-3
    if kind == "constant":         # 0.1: ends in a set bit pattern that ties at whole binades
        return np.full(shape, 0.1)
    if kind == "dyadic":
        return np.where(rng.random(shape) < 0.5, 1.0, 0.125)
    if kind == "wide":             # forty binades, zeros and negative cells among them
        return np.exp(rng.uniform(-30, 0, shape)) * rng.choice([1.0, 1.0, 0.0, -1.0], shape)
    if kind == "star":
        x = np.meshgrid(*[np.linspace(-1, 1, n) for n in shape], indexing="ij", sparse=True)
        return np.maximum(1e-6, 1 - 4 * sum(v * v for v in x)) * np.exp(0.01 * rng.standard_normal(shape))
    if kind == "tiny":             # below the binades the records cover
        return rng.random(shape) * 1e-305
    if kind == "huge":
        r = rng.random(shape)
        r[1, 1, 1] = 1e300
        return r
    raise ValueError(kind)


# fewer cells than a run, one group and a bit, odd rows, just above two super-groups, many groups
@pytest.mark.parametrize("shape", [(3, 3, 3), (10, 11, 10), (23, 31, 29), (41, 40, 41), (70, 66, 72)])
@pytest.mark.parametrize("kind", ["random", "constant", "dyadic", "wide", "star", "tiny", "huge"])
@pytest.mark.parametrize("box", [UNIT, CENTRED])
def test_sequential_moments_bitwise(kind, shape, box):
    rho = density(kind, shape)
    o = OracleSim(*shape, lo=box[0], hi=box[1], G=1.0)
    with hc.HydroSolver3D(shape, lo=box[0], hi=box[1], G=1.0, gravity_only=1, max_iter=1, tol=1e-30) as s:
        s.gravity_solve(rho)
        got = s.moments()
    want = o.moments_ref(rho)
    assert np.array_equal(got, want, equal_nan=True), (got - want, got, want)
