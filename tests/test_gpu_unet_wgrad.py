"""Weight gradients of the network's convolutions at the edges of both kernels:
rows that one or two CTAs share, planes of one row, volumes of one plane, rows
as long as the row kernel's shared memory allows and longer.  Small whole
numbers make every product and sum exact in FP32, so the result is compared
for equality."""
import ctypes as C

import numpy as np
import pytest
import torch

import hydrocode_astro1_b200 as hc

pytestmark = pytest.mark.gpu


def _bits(a):
    return torch.from_numpy(a.astype(np.float32)).to(torch.bfloat16).view(torch.int16).numpy().view(np.uint16).copy()


def _ptr(a, t):
    return a.ctypes.data_as(C.POINTER(t))


@pytest.mark.parametrize("shape,parts", [
    ((3, 5, 48), 1), ((3, 5, 48), 3), ((5, 1, 64), 1), ((1, 16, 48), 2), ((2, 2, 128), 1), ((4, 9, 144), 2),
    ((3, 20, 272), 3), ((2, 6, 512), 1), ((2, 6, 528), 1), ((3, 7, 40), 2), ((6, 40, 16), 5), ((64, 48, 64), 148),
])
def test_weight_gradient_exact(shape, parts):
    rng = np.random.default_rng(sum(shape) + parts)
    n = int(np.prod(shape))
    x, dy = (rng.integers(-4, 5, (n, 16)) for _ in range(2))   # sums below 16 n < 2^24
    dw = np.zeros((16, 27, 16), np.float32)
    assert hc.lib().hc_unet_wgrad_test(*shape, _ptr(_bits(x), C.c_uint16), _ptr(_bits(dy), C.c_uint16), parts,
                                       _ptr(dw, C.c_float)) == 0
    pad = np.zeros([s + 2 for s in shape] + [16], np.int64)
    pad[1:-1, 1:-1, 1:-1] = x.reshape(*shape, 16)
    ref = np.empty((16, 27, 16), np.int64)
    for t in range(27):
        a, b, c = t // 9, t // 3 % 3, t % 3
        ref[:, t] = dy.T @ pad[a:a + shape[0], b:b + shape[1], c:c + shape[2]].reshape(n, 16)
    assert np.array_equal(dw, ref)
