"""The loss and its gradient against the FP64 oracle at image sizes on both sides of the kernels' tiles (32 x 32
and a halo of 5, staged as 32 columns and 10), and the value without a gradient.

Tolerances as in test_gpu_backward.py: value 1e-5 absolute, dL/drgb 1e-4 of its largest entry."""
import ctypes as C

import numpy as np
import pytest

import oracle
import webgs

pytestmark = pytest.mark.gpu
LAMBDA = 0.2


@pytest.mark.parametrize("w,h", [(1, 1), (2, 7), (5, 16), (11, 33), (26, 27), (27, 26), (31, 64), (32, 32), (33, 31), (37, 5),
                                 (59, 65), (3, 200), (400, 2)])
def test_loss_sizes(gpu_ctx, w, h):
    rng = np.random.default_rng(1000 * w + h)
    x = rng.uniform(0, 1, (h, w, 3)).astype(np.float32)
    y = np.clip(x + rng.normal(0, 0.1, x.shape), 0, 1).astype(np.float32)
    val, dl = gpu_ctx.loss(x, y, LAMBDA)
    rval, rdl = oracle.loss_l1_ssim(x, y, LAMBDA)
    assert abs(val - rval) < 1e-5
    assert np.abs(dl - rdl).max() <= 1e-4 * np.abs(rdl).max()
    only = C.c_double()
    rc = webgs.library().gs_loss_l1_ssim(gpu_ctx.handle, x.ctypes.data, y.ctypes.data, w, h, LAMBDA, C.byref(only), None, 0)
    assert rc == 0 and only.value == val
