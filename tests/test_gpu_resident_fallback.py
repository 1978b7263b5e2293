"""The way back from the resident SOR launch: a launch that is refused, or whose
blocks give up waiting for one another, leaves the solve to the separate sweeps
with the same potential, iteration count and norm, bit for bit, and later solves
too.  Two contexts that relax at the same time on threads of their own give what
they give alone."""
import threading

import numpy as np
import pytest

import hydrocode_astro1_b200 as hc

pytestmark = pytest.mark.gpu

REFUSED, GAVE_UP = 1, 2


def problem(shape, seed):
    rng = np.random.default_rng(seed)
    return rng.random(shape) + 0.1, rng.standard_normal(shape)


def solve(s, rho, state):
    if state:
        q = np.zeros((5,) + rho.shape)
        q[0], q[4] = rho, 1.0
        s.set_state(q)
    rc = s.gravity_solve(None if state else rho)
    d = s.diagnostics()
    return s.phi(), (rc, d["last_iterations"], d["last_residual"], d["outer_cycles"])


def two_solves(shape, fault, **kw):
    rho, phi = problem(shape, 1)
    with hc.HydroSolver3D(shape, G=1.0, moment_order=hc.MOMENTS_TREE, **kw) as s:
        assert hc.lib().hc_resident_fault(s.h, fault) == hc.HC_OK
        s.set_phi(phi)
        first = solve(s, rho, not kw.get("gravity_only"))
        assert hc.lib().hc_resident_fault(s.h, 0) == hc.HC_OK
        second = solve(s, rho * 1.5, not kw.get("gravity_only"))
        launches = s.timing()["sor_launches"]
    return first, second, launches


def same(a, b):
    return np.array_equal(a[0], b[0]) and a[1] == b[1]


@pytest.mark.parametrize("shape", [(20, 18, 22), (33, 40, 31), (90, 101, 97)])
@pytest.mark.parametrize("kw", [dict(grav_bc=1), dict(grav_bc=1, lmax=4), dict(grav_bc=0), dict(grav_bc=2)])
@pytest.mark.parametrize("fault", [REFUSED, GAVE_UP])
def test_fp64_solve_again(shape, kw, fault):
    kw = dict(kw, gravity_only=1, max_iter=3000, tol=1e-5)
    plain, mended = two_solves(shape, 0, **kw), two_solves(shape, fault, **kw)
    assert same(plain[0], mended[0]) and same(plain[1], mended[1])
    assert mended[2] > 10 * plain[2]      # the sweeps ran separately


@pytest.mark.parametrize("shape", [(20, 18, 22), (64, 60, 64), (61, 50, 99)])
@pytest.mark.parametrize("fault", [REFUSED, GAVE_UP])
def test_mixed_solve_again(shape, fault):
    kw = dict(precision=hc.FP32, max_iter=20000, tol=1e-6)
    plain, mended = two_solves(shape, 0, **kw), two_solves(shape, fault, **kw)
    assert same(plain[0], mended[0]) and same(plain[1], mended[1])
    assert mended[2] > 2 * plain[2]


@pytest.mark.parametrize("precision", [hc.FP64, hc.FP32])
def test_two_contexts_at_once(precision):
    shapes = [(128, 120, 128), (96, 90, 100)]

    def run(k, got):
        shape = shapes[k]
        rho, _ = problem(shape, k)
        with hc.HydroSolver3D(shape, G=1.0, moment_order=hc.MOMENTS_TREE, precision=precision, tol=1e-5,
                              max_iter=20000) as s:
            for r in range(6):
                got[k].append(solve(s, rho * (1.0 + 0.1 * r), True))

    alone, together = [[], []], [[], []]
    for k in range(2):
        run(k, alone)
    threads = [threading.Thread(target=run, args=(k, together)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(2):
        assert len(together[k]) == 6
        for a, b in zip(alone[k], together[k]):
            assert same(a, b)
