"""A frame that is refused for memory takes the context's last frame with it: some of its buffers are replaced by
then. Its gradient is refused (it would read buffers that are gone), and the next frames are as ever."""
import numpy as np
import pytest

import webgs
from webgs import _abi
from webgs import workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [False, True])
def test_no_gradient_after_a_frame_that_did_not_fit(batch):
    small, large, factor = 10, 4000, 1_000_000  # 40 MB and 16 GB for each of the four key and value buffers
    view = W.CameraSpec((0.0, 0.0, -4.0), (0, 0, 0), 60.0, 96, 80).view()
    packed = W.SceneSpec(small, 3, 0).build()
    packed[3 * small:6 * small] += 2.0
    dl = np.random.default_rng(1).normal(0.0, 1e-3, (80, 96, 3)).astype(np.float32)
    with webgs.Context(flags=webgs.GS_FLAG_DIFFERENTIABLE, max_instance_factor=factor) as ctx:
        a, b = ctx.upload(packed, small), ctx.upload(W.SceneSpec(large, 4, 0).build(), large)

        def forward(sc):
            if batch:
                return ctx.forward_batch([(sc, view)], rgba8=False, rgb=True)[0]["rgb"]
            return ctx.forward(sc, view, rgba8=False, rgb=True)["rgb"]

        def backward(sc):
            return ctx.backward_batch(sc, [dl]) if batch else ctx.backward(sc, dl)

        rgb = forward(a)
        want = backward(a)
        assert np.abs(want).max() > 0.0
        held = [torch.empty(torch.cuda.mem_get_info()[0] - (24 << 30), dtype=torch.uint8, device="cuda")]
        with pytest.raises(webgs.GsError) as refused:
            forward(b)
        assert refused.value.code in (_abi.GS_ERR_OOM, _abi.GS_ERR_CUDA)
        with pytest.raises(webgs.GsError) as gone:
            backward(a)
        assert gone.value.code == _abi.GS_ERR_STATE
        held.clear()
        torch.cuda.empty_cache()
        np.testing.assert_array_equal(forward(a), rgb)
        assert np.abs(backward(a) - want).max() <= 1e-5 * np.abs(want).max()
        a.close()
        b.close()
