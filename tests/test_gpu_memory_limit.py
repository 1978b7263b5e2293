"""A solve that the device memory just holds runs, although the work memory that
only makes its moments faster was taken first: that is given back."""
import numpy as np
import pytest

import hydrocode_astro1_b200 as hc

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
MIB = 1 << 20


@pytest.mark.skipif(not torch.cuda.is_available(), reason="no CUDA device")
def test_faster_buffers_give_way():
    shape = (256, 256, 256)      # split potential and density: 128 MiB each
    rho = np.random.default_rng(0).random(shape) + 0.1

    def solve(fill):
        with hc.HydroSolver3D(shape, G=1.0, gravity_only=1, tol=1e-30) as s:
            s.set_gravity_params(1.5, 0, 1e-30)
            s.gravity_solve(rho)                       # moments alone: their work memory is taken
            free, _ = torch.cuda.mem_get_info()
            block = torch.empty(free - 236 * MIB, dtype=torch.uint8, device="cuda") if fill else None
            s.set_gravity_params(1.5, 4, 1e-30)
            s.gravity_solve(rho)
            phi = s.phi()
            del block
            torch.cuda.empty_cache()
        return phi

    assert np.array_equal(solve(True), solve(False))


@pytest.mark.skipif(not torch.cuda.is_available(), reason="no CUDA device")
@pytest.mark.parametrize("precision,later", [(hc.FP32, 0), (hc.FP64, 2 * 128 ** 3 * 8)])
def test_first_solve_finds_its_buffers(precision, later):
    """All but the FP64 split fields are there before the first solve."""
    shape = (128, 128, 128)
    q = np.zeros((5,) + shape)
    q[0], q[4] = np.random.default_rng(0).random(shape) + 0.1, 1.0

    def taken():
        with hc.HydroSolver3D(shape, G=1.0, tol=1e-4, precision=precision) as s:
            s.set_state(q)
            before, _ = torch.cuda.mem_get_info()
            s.gravity_solve()
            return before - torch.cuda.mem_get_info()[0]

    taken()                                            # loads the kernels
    assert taken() <= later
