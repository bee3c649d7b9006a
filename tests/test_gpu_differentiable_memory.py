"""A differentiable context's frame takes no more device memory than a plain one's, beyond what grows with the
image alone: at most a word per tile and 8x4 block. And its gradients do not depend on which of the sort's buffers
held the values last: a frame of an odd number of sort passes gives those of an even number's."""
import numpy as np
import pytest

import oracle
import webgs
from test_gpu_backward import _compare
from webgs import workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [8, 16, 32])
def test_a_differentiable_frame_needs_no_more_memory(tile):
    spec, cam = W.SceneSpec(1_000_000, 2, 1, 64, 20.0), W.CAMERA_1080P
    packed, used = spec.build(), []
    for flags in (webgs.GS_FLAG_DIFFERENTIABLE, 0, webgs.GS_FLAG_DIFFERENTIABLE):  # the first loads the kernels too
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        with webgs.Context(flags=flags, tile_size=tile) as ctx:
            sc = ctx.upload(packed, spec.count)
            ctx.forward(sc, cam.view())
            used.append(before - torch.cuda.mem_get_info()[0])
            sc.close()
    blocks = 1920 * 1088 // 32
    assert used[2] - used[1] <= 4 * blocks + (4 << 20), used  # the allocator's pages are 2 MiB


@pytest.mark.parametrize("tile", [8, 16, 32])
@pytest.mark.parametrize("digit_bits,size", [(8, (16, 16)), (8, (96, 80)), (4, (96, 80)), (4, (40, 24))])
@pytest.mark.parametrize("n", [1, 40, 3000])
def test_gradients_after_any_number_of_passes(n, digit_bits, size, tile):
    w, h = size
    packed = W.SceneSpec(n, 50 + n, 0).build()
    packed[:3] = (0.05, 0.02, 0.0)
    packed[3 * n:6 * n] += 1.0
    view = W.CameraSpec((0.1, 0.2, -4.0), (0, 0, 0), 60.0, w, h).view()
    dl = np.random.default_rng(n).normal(0.0, 1e-3, (h, w, 3)).astype(np.float32)
    with webgs.Context(flags=webgs.GS_FLAG_DIFFERENTIABLE, tile_size=tile, digit_bits=digit_bits) as ctx:
        sc = ctx.upload(packed, n)
        for _ in range(2):
            ctx.forward(sc, view, rgba8=False, rgb=True)
            got = ctx.backward(sc, dl)
        sc.close()
    want, _ = oracle.backward_f64(webgs.view_bytes(view), packed, n, dl, tile=tile)
    _compare(got, want, n)
