"""Views of one scene that share a launch per stage (eight or more small views): sizes whose keys take different
numbers of sort passes, from one tile up, and outputs that differ from view to view, over every tile size and
digit width. Each view has to equal its single frame bit for bit, the first time and on a graph's replay."""
import pytest

import webgs
from webgs import _abi
from webgs import workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIZES = ((96, 64), (16, 8), (641, 479), (250, 1), (128, 333))
OUTPUTS = (("rgba8",), ("rgb", "final_t"), ("rgba8", "rgb", "final_t", "n_contrib"))


def _buffers(names, w, h):
    made = {"rgba8": lambda: torch.zeros(h, w, 4, dtype=torch.uint8, device="cuda"),
            "rgb": lambda: torch.zeros(h, w, 3, device="cuda"),
            "final_t": lambda: torch.zeros(h, w, device="cuda"),
            "n_contrib": lambda: torch.zeros(h, w, dtype=torch.int32, device="cuda")}
    return {k: made[k]() for k in names}


@pytest.mark.parametrize("tile,digit_bits,sort_block,views,n", [
    (16, 8, 4096, 17, 20_000), (8, 4, 2048, 8, 20_000), (32, 8, 2048, 9, 5_000), (16, 8, 4096, 7, 5_000),
    (16, 8, 4096, 16, 1), (8, 8, 4096, 12, 60_000)])
def test_runs_equal_single_frames(tile, digit_bits, sort_block, views, n):
    spec = W.SceneSpec(n, 4, 1, 64, 20.0)
    cams = [W.orbit_cameras(1, k, 9.0, fixed_resolution=SIZES[k % 5])[0][1].view() for k in range(views)]
    with webgs.Context(tile_size=tile, digit_bits=digit_bits, sort_block=sort_block) as ctx:
        sc = ctx.upload(spec.build(), n)
        out = [_buffers(OUTPUTS[k % 3], *SIZES[k % 5]) for k in range(views)]
        items = (_abi.BatchView * views)()
        for item, view, bufs in zip(items, cams, out):
            p = {k: t.data_ptr() for k, t in bufs.items()}
            item.scene, item.view = sc.handle, view
            item.out = _abi.Image(webgs.GS_MEM_DEVICE, p.get("rgba8"), p.get("rgb"), p.get("final_t"), p.get("n_contrib"))
        torch.cuda.synchronize()
        for _ in range(3):
            assert webgs.library().gs_forward_batch(ctx.handle, items, views) == _abi.GS_OK
            ctx.synchronize()
            got = [{k: t.clone() for k, t in bufs.items()} for bufs in out]
            for bufs in out:
                for t in bufs.values():
                    t.fill_(7)
            torch.cuda.synchronize()
        for k, view in enumerate(cams):
            want = _buffers(OUTPUTS[k % 3], *SIZES[k % 5])
            ctx.forward_device(sc, view, **{name: t.data_ptr() for name, t in want.items()})
            ctx.synchronize()
            for name, t in want.items():
                assert torch.equal(got[k][name].view(torch.uint8), t.view(torch.uint8)), (k, name)
        sc.close()
