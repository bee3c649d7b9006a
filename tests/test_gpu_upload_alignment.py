"""Uploads from device buffers at every offset within 16 bytes, for scene sizes that put each attribute block
and its end anywhere within 16 bytes too, and on both sides of the transpose's 128 Gaussians: the frame's
intermediates (means, covariances, colours) equal the oracle's bit for bit."""
import numpy as np
import pytest

import webgs
from helpers import assert_frame_parity, gpu_frame, oracle_frame
from webgs import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 5, 63, 64, 65, 127, 128, 129, 130, 255, 257, 1003])
def test_device_buffers_at_any_offset(gpu_ctx, n):
    torch = pytest.importorskip("torch")
    packed = W.SceneSpec(n, 50 + n, 0).build()
    view = W.CameraSpec((0.0, 0.0, -4.0), (0.0, 0.0, 0.0), 60.0, 40, 32).view()
    o = oracle_frame(view, packed, n)
    for offset in range(4):
        buf = torch.full((59 * n + 8,), float("nan"), device="cuda")
        buf[offset:offset + 59 * n] = torch.from_numpy(packed).cuda()
        torch.cuda.synchronize()
        sc = gpu_ctx.upload(buf.data_ptr() + 4 * offset, n, webgs.GS_MEM_DEVICE)
        assert_frame_parity(gpu_frame(gpu_ctx, sc, view), o)
        sc.update(np.zeros_like(packed))
        sc.update(buf.data_ptr() + 4 * offset, webgs.GS_MEM_DEVICE)
        assert_frame_parity(gpu_frame(gpu_ctx, sc, view), o)
        sc.close()
