"""The raster backward's reduction of hits (staged 64 at a time, summed eight at a time over an 8x4 block)
against the FP64 adjoint, at list lengths on both sides of 8, 32 and 64, odd image sizes and every tile
size; and a pixel whose dL/drgb is not finite, which must not reach Gaussians it does not blend.

Tolerances as in test_gpu_backward.py (fp32 sums and T recovered by division): per parameter group
||g32 - g64|| <= 2e-3 ||g64||; two runs of the same sums in another order agree to 1e-5 of the largest."""
import numpy as np
import pytest

import oracle
import webgs
from test_gpu_backward import _compare
from webgs import workloads as W

pytestmark = pytest.mark.gpu


def _scene(n, seed):
    packed = W.SceneSpec(n, seed, 0).build()
    packed[3 * n:6 * n] += 2.5  # splats of about 8 pixels: every block of the image meets most of them
    return packed


@pytest.mark.parametrize("tile", [8, 16, 32])
@pytest.mark.parametrize("n", [2, 7, 8, 9, 31, 33, 64, 65, 200])
def test_list_lengths(n, tile):
    packed = _scene(n, 100 + n)
    view = W.CameraSpec((0.1, 0.2, -4.0), (0, 0, 0), 60.0, 101, 67).view()
    dl = np.random.default_rng(n).normal(0.0, 1e-3, (67, 101, 3)).astype(np.float32)
    with webgs.Context(flags=webgs.GS_FLAG_DIFFERENTIABLE, tile_size=tile) as ctx:
        sc = ctx.upload(packed, n)
        ctx.forward(sc, view, rgba8=False, rgb=True)
        g32 = ctx.backward(sc, dl)
        sc.close()
    g64, _ = oracle.backward_f64(webgs.view_bytes(view), packed, n, dl, tile=tile)
    _compare(g32, g64, n)


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_a_pixel_without_a_finite_gradient(bad):
    n = 400
    packed = W.SceneSpec(n, 77, 0).build()
    view = W.CameraSpec((0.0, 0.0, -4.0), (0, 0, 0), 60.0, 96, 96).view()
    dl = np.random.default_rng(5).normal(0.0, 1e-3, (96, 96, 3)).astype(np.float32)
    dl[48, 47] = 0.0
    with webgs.Context(flags=webgs.GS_FLAG_DIFFERENTIABLE) as ctx:
        sc = ctx.upload(packed, n)
        ctx.forward(sc, view, rgba8=False, rgb=True)
        zero = ctx.backward(sc, dl)
        dl[48, 47, 1] = bad
        g = ctx.backward(sc, dl)
        again = ctx.backward(sc, np.where(np.isfinite(dl), dl, 0.0).astype(np.float32))
        sc.close()
    logits, rest = slice(13 * n, 14 * n), g[14 * n:].reshape(n, 45)
    touched = ~np.isfinite(rest).all(1)  # Gaussians that the pixel blends
    assert 0 < touched.sum() < n // 2
    assert np.abs(g[logits] - zero[logits])[~touched].max() <= 1e-5 * np.abs(zero[logits]).max()
    scale = np.abs(zero[14 * n:]).max()
    assert np.abs(rest - zero[14 * n:].reshape(n, 45))[~touched].max() <= 1e-5 * scale
    assert np.abs(again - zero).max() <= 1e-5 * np.abs(zero).max()
