"""A context makes a graph for the second frame in a row of one scene, size and set of outputs and replays it from
then on; every other frame is launched as it is. Whatever order frames come in, each has to be its own: another
scene, size or set of outputs between two replays, back and forth, new values and views under a graph, a scene
destroyed and another in its place (an address that comes back), batches and gradients in between, a frame that
is refused."""
import numpy as np
import pytest

import webgs
from webgs import workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SIZES = {"small": (96, 64), "wide": (250, 30), "large": (320, 240)}
SCENES = {"a": (4_000, 1), "b": (4_000, 2), "c": (9_000, 3)}
OUTPUTS = {"8": ("rgba8",), "f": ("rgb", "final_t"), "all": ("rgba8", "rgb", "final_t", "n_contrib")}


def _view(size, k=0):
    return W.CameraSpec((0.1 * k, 0.2, -4.0), (0.0, 0.0, 0.0), 60.0, *SIZES[size]).view()


def _packed(scene):
    return W.SceneSpec(*SCENES[scene], 0).build()


def _buffers(size, outputs):
    w, h = SIZES[size]
    shape = {"rgba8": ((h, w, 4), torch.uint8), "rgb": ((h, w, 3), torch.float32), "final_t": ((h, w), torch.float32),
             "n_contrib": ((h, w), torch.int32)}
    return {k: torch.full(shape[k][0], 7, dtype=shape[k][1], device="cuda") for k in OUTPUTS[outputs]}


def _want(cache, scene, size, k):
    key = (scene, size, k)
    if key not in cache:
        with webgs.Context(flags=webgs.GS_FLAG_NO_GRAPH) as ctx:
            sc = ctx.upload(_packed(scene), SCENES[scene][0])
            cache[key] = ctx.forward(sc, _view(size, k), rgba8=True, rgb=True, final_t=True, n_contrib=True)
            sc.close()
    return cache[key]


@pytest.fixture(scope="module")
def wants():
    return {}


def _frame(ctx, scenes, wants, buffers, scene, size, outputs, k):
    bufs = buffers.setdefault((size, outputs), _buffers(size, outputs))
    for t in bufs.values():
        t.fill_(7)
    torch.cuda.synchronize()
    ctx.forward_device(scenes[scene], _view(size, k), **{name: t.data_ptr() for name, t in bufs.items()})
    ctx.synchronize()
    for name, t in bufs.items():
        want = _want(wants, scene, size, k)[name]
        np.testing.assert_array_equal(t.cpu().numpy().view(np.uint8), np.ascontiguousarray(want).view(np.uint8),
                                      err_msg=str((scene, size, outputs, k, name)))


SEQUENCES = {
    "a key between two replays": [("a", "small", "8")] * 4 + [("a", "large", "8")] + [("a", "small", "8")] * 2,
    "a second graph between": [("a", "small", "8")] * 3 + [("b", "wide", "f")] * 3 + [("a", "small", "8")] * 3,
    "by turns": [("a", "small", "8"), ("b", "small", "8")] * 4,
    "pairs by turns": ([("a", "small", "8")] * 2 + [("b", "small", "8")] * 2) * 3,
    "other outputs": [("a", "small", "8")] * 3 + [("a", "small", "all")] * 3 + [("a", "small", "f"), ("a", "small", "8")] * 2,
    "buffers grow under a graph": [("a", "small", "8")] * 3 + [("c", "large", "all")] * 2 + [("a", "small", "8")] * 3,
}


@pytest.mark.parametrize("name", SEQUENCES)
def test_frames_in_any_order(name, wants):
    with webgs.Context() as ctx:
        scenes = {s: ctx.upload(_packed(s), SCENES[s][0]) for s in SCENES}
        buffers = {}
        for k, (scene, size, outputs) in enumerate(SEQUENCES[name]):
            _frame(ctx, scenes, wants, buffers, scene, size, outputs, k % 3)
        for sc in scenes.values():
            sc.close()


def test_random_orders(wants):
    rng = np.random.default_rng(4)
    with webgs.Context() as ctx:
        scenes = {s: ctx.upload(_packed(s), SCENES[s][0]) for s in SCENES}
        buffers = {}
        for _ in range(60):
            key = (rng.choice(list(SCENES)), rng.choice(list(SIZES)), rng.choice(list(OUTPUTS)))
            for _ in range(int(rng.integers(1, 4))):
                _frame(ctx, scenes, wants, buffers, *key, int(rng.integers(0, 3)))
        for sc in scenes.values():
            sc.close()


def test_a_scene_in_a_destroyed_ones_place(wants):
    with webgs.Context() as ctx:
        buffers = {}
        for scene in ("a", "b", "a", "b", "c", "a"):  # same size: the allocations come back at their addresses
            sc = ctx.upload(_packed(scene), SCENES[scene][0])
            for k in range(3):
                _frame(ctx, {scene: sc}, wants, buffers, scene, "small", "8", k)
            sc.close()


def test_new_values_under_a_graph(wants):
    with webgs.Context() as ctx:
        sc, buffers = ctx.upload(_packed("a"), SCENES["a"][0]), {}
        for scene in ("a", "b", "a", "a", "b"):
            sc.update(_packed(scene))
            for k in range(3):
                _frame(ctx, {scene: sc}, wants, buffers, scene, "small", "8", k)
        sc.close()


def test_batches_refusals_and_gradients_between(wants):
    with webgs.Context(flags=webgs.GS_FLAG_DIFFERENTIABLE) as ctx:
        scenes = {s: ctx.upload(_packed(s), SCENES[s][0]) for s in SCENES}
        buffers, grads = {}, {}
        dl = np.random.default_rng(2).normal(0.0, 1e-3, (64, 96, 3)).astype(np.float32)
        for turn in range(3):
            for scene in ("a", "a", "a", "b"):
                _frame(ctx, scenes, wants, buffers, scene, "small", "all", 1)
                g = ctx.backward(scenes[scene], dl)
                ref = grads.setdefault(scene, g)
                assert np.abs(g - ref).max() <= 1e-5 * np.abs(ref).max()
            out = ctx.forward_batch([(scenes["a"], _view("small", 2)), (scenes["b"], _view("wide", 0)), (scenes["a"], _view("small", 0))])
            for o, (scene, size, k) in zip(out, (("a", "small", 2), ("b", "wide", 0), ("a", "small", 0))):
                np.testing.assert_array_equal(o["rgba8"], _want(wants, scene, size, k)["rgba8"])
            bad = _view("small")
            bad.texture_size[0] = 0.0
            with pytest.raises(webgs.GsError):
                ctx.forward_device(scenes["a"], bad, rgba8=buffers[("small", "all")]["rgba8"].data_ptr())
        for sc in scenes.values():
            sc.close()
