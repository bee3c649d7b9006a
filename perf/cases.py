"""The work that users of the splat pipeline have it do, as cases that can be timed and compared.

Every case goes through the public entry points (webgs.Renderer, webgs.Context, and the C ABI of
include/gs.h where a training loop passes device buffers). The kinds, and what each stands for:

  viewer       an interactive viewer: Renderer.execute() after each mouse move, image on the host
  frame        one frame of one scene into device buffers, as an offline renderer or an encoder takes it
  closeup      a frame from inside a small scene: few splats, each over a large part of the image
  mixed        one context that renders views of different sizes in turn (an evaluation set)
  batch        views of several scenes in one gs_forward_batch
  turntable    small views of one scene by gs_forward_batch_cameras (thumbnails of an orbit)
  train        an optimizer's step: new attributes into the scene, forward, loss, backward, on the device
  train_batch  the same with several views per step, their gradients summed
  loss         L1 + SSIM of two images with its gradient and its value (a metric, or a 2D fit)

Scenes have the distributions of the benchmark configurations (a unit cluster, or a mixture of
anisotropic clusters in a box; log-scales about -4, opacity logits N(0, 1.5^2), degree-3 SH), made on
the GPU from the seed. The views differ with the seed too.
"""
import ctypes as C
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parent.parent / "web-gs-renderer_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import webgs  # noqa: E402
from webgs import _abi  # noqa: E402

DEV = "cuda"
RESOLUTIONS = ((640, 480), (1280, 720), (1920, 1080))  # what batches of views are drawn from
NEAR, FAR = 0.2, 1000.0
LAMBDA = 0.2  # weight of the SSIM term


# ---- the cases -------------------------------------------------------------------------------------
def _case(name, kind, n, width, height, **more):
    c = {"name": name, "kind": kind, "n": n, "width": width, "height": height, "views": 1, "tile": 16,
         "digit_bits": 8, "raster_batch": 256, "sort_block": 4096, "outputs": "rgba8"}
    c.update(more)
    return c


def listed():
    return [
        # the smallest interactive frame: the 50k configuration, image in ordinary host memory
        _case("viewer_50k_512", "viewer", 50_000, 512, 512),
        # the headline configuration: one frame of 1M Gaussians at 1920x1080
        _case("frame_1m_1080p", "frame", 1_000_000, 1920, 1080),
        # the largest single frame: 3M Gaussians at 4K, with the fp32 colours kept
        _case("frame_3m_4k", "frame", 3_000_000, 3840, 2160, outputs="rgba8,rgb"),
        # an odd size with 8x8 tiles and every output, as compositing and debugging ask for
        _case("frame_250k_odd_tile8", "frame", 250_003, 1237, 823, tile=8, outputs="rgb,final_t,n_contrib"),
        # a camera in the middle of the splats: each covers many tiles
        _case("closeup_60k_900p", "closeup", 60_000, 1600, 900, outputs="rgb,final_t"),
        # an evaluation set: six views of three sizes through one context
        _case("mixed_400k_6_views", "mixed", 400_000, 1920, 1080, views=6),
        # the batched configuration: 16 views of scenes of 100k, 400k and 1.5M, in the tile size that the
        # autotuner picks for it
        _case("batch_16_views", "batch", 1_500_000, 1920, 1080, views=16, tile=32),
        # thumbnails of a turntable from cameras
        _case("turntable_24_100k", "turntable", 100_000, 320, 240, views=24),
        # an early training step: few Gaussians, a small odd photograph, the loss read every step
        _case("train_20k_397x301", "train", 20_011, 397, 301),
        # the differentiation configuration: 500k Gaussians at 1280x720
        _case("train_500k_720p", "train", 500_000, 1280, 720),
        # the batched differentiation configuration: one 3M scene, eight views at 1920x1080
        _case("train_8_views_3m", "train_batch", 3_000_000, 1920, 1080, views=8),
        # the loss alone on full-size images
        _case("loss_1080p", "loss", 0, 1920, 1080),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["viewer", "frame", "frame", "closeup", "mixed", "batch", "turntable", "train", "train",
                       "train_batch", "loss"])
    options = {"tile": rng.choice([16, 16, 16, 32, 8]), "digit_bits": rng.choice([8, 8, 8, 4]),
               "raster_batch": rng.choice([256, 256, 128, 64, 32]), "sort_block": rng.choice([4096, 4096, 2048])}
    views = 1
    if kind == "viewer":
        n, w, h = _log(rng, 2_000, 400_000), _log(rng, 96, 1920), _log(rng, 96, 1080)
        options["outputs"] = "rgba8"
    elif kind == "frame":
        n, w, h = _log(rng, 2_000, 3_000_000), _log(rng, 64, 3840), _log(rng, 64, 2160)
        options["outputs"] = rng.choice(["rgba8", "rgba8", "rgb", "rgba8,rgb", "rgb,final_t,n_contrib"])
        if options["tile"] == 8:  # at most 65536 tiles fit a key
            w, h = min(w, 1920), min(h, 1080)
    elif kind == "closeup":
        n, w, h = _log(rng, 2_000, 60_000), _log(rng, 64, 1600), _log(rng, 64, 900)
        options["outputs"] = rng.choice(["rgba8", "rgb,final_t"])
    elif kind in ("mixed", "batch"):
        n, w, h = _log(rng, 15_000, 1_500_000), 1920, 1080
        views = rng.randint(3, 6) if kind == "mixed" else rng.randint(2, 16)
    elif kind == "turntable":
        n, w, h, views = _log(rng, 2_000, 200_000), _log(rng, 64, 640), _log(rng, 64, 480), rng.randint(2, 24)
    elif kind == "train":
        n, w, h = _log(rng, 2_000, 1_000_000), _log(rng, 64, 1920), _log(rng, 48, 1080)
    elif kind == "train_batch":
        n, w, h, views = _log(rng, 2_000, 1_000_000), _log(rng, 64, 1920), _log(rng, 48, 1080), rng.randint(2, 4)
    else:
        n, w, h = 0, _log(rng, 16, 3840), _log(rng, 16, 2160)
    c = _case("", kind, n, w, h, views=views, **options)
    del c["name"]
    return c


# ---- inputs ----------------------------------------------------------------------------------------
def _generator(seed, stream):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 7919 + stream)
    return g


def _unit_quats(n, g):
    q = torch.randn(n, 4, generator=g, device=DEV)
    return q / q.norm(dim=1, keepdim=True)


def _box(n):
    """Edge of the scene's box: 20 at a million Gaussians, the density kept for other counts."""
    return 20.0 * max(n / 1e6, 0.02) ** (1.0 / 3.0)


def _scene(n, seed, mixture, log_scale=-4.0):
    """A scene in the packed layout (59 n floats): positions, log-scales, rotations, DC, opacity, rest."""
    g = _generator(seed, 1)
    pos = torch.randn(n, 3, generator=g, device=DEV)
    if mixture:
        clusters, box = 64, _box(n)
        centre = (torch.rand(clusters, 3, generator=g, device=DEV) - 0.5) * box
        sigma = (0.3 + 2.2 * torch.rand(clusters, 3, generator=g, device=DEV)) * (box / 20.0)
        w, x, y, z = _unit_quats(clusters, g).unbind(1)
        rot = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                           2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                           2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).view(-1, 3, 3)
        pick = torch.randint(clusters, (n,), generator=g, device=DEV)
        a = pos * sigma[pick]
        turned = torch.stack([(rot[pick, r] * a).sum(1) for r in range(3)], 1)
        pos = (centre[pick] + turned).clamp(-box / 2, box / 2)
    scale = log_scale + 0.5 * torch.randn(n, 3, generator=g, device=DEV)
    quat = _unit_quats(n, g)
    dc = 0.5 * torch.randn(n, 3, generator=g, device=DEV)
    logit = 1.5 * torch.randn(n, generator=g, device=DEV)
    rest = 0.05 * torch.randn(n, 45, generator=g, device=DEV)
    return torch.cat([t.reshape(-1) for t in (pos, scale, quat, dc, logit, rest)])


def _photo(width, height, seed):
    """An image that a training step is fitted to: smooth structure, fine texture, values in [0, 1]."""
    g = _generator(seed, 2)
    img = torch.zeros(1, 3, height, width, device=DEV)
    for cells, weight in ((4, 0.5), (16, 0.3), (64, 0.15)):
        coarse = torch.rand(1, 3, min(cells, height), min(cells, width), generator=g, device=DEV)
        img += weight * torch.nn.functional.interpolate(coarse, (height, width), mode="bilinear", align_corners=False)
    img += 0.05 * torch.rand(1, 3, height, width, generator=g, device=DEV)
    return img[0].permute(1, 2, 0).contiguous()


def _scene_counts(case):
    """Gaussian counts of a case's scenes: the batch has three of them, as 1.5M : 400k : 100k."""
    n = case["n"]
    return [n, max(1, n * 4 // 15), max(1, n // 15)] if case["kind"] == "batch" else [n]


def _f32(values):
    return tuple(float(np.float32(v)) for v in values)


def _cameras(case, seed):
    """(scene slot, eye, target, vertical field of view, width, height) of each view."""
    rng, plan = np.random.default_rng(seed * 31 + 5), np.random.default_rng(8)
    kind, w, h = case["kind"], case["width"], case["height"]
    counts = _scene_counts(case)
    out = []
    for v in range(case["views"]):
        slot = int(plan.integers(len(counts)))  # scenes and sizes belong to the case, not to the seed
        box = _box(counts[slot])
        if kind == "closeup":
            eye, target, fov = rng.normal(0, 0.15, 3), rng.normal(0, 0.3, 3) + (0, 0, 1.5), 70.0
        elif kind == "turntable":
            a = 2 * math.pi * (v + rng.uniform()) / case["views"]
            eye, target, fov = (4.5 * math.sin(a), 0.8, 4.5 * math.cos(a)), (0, 0, 0), 50.0
        elif case["views"] > 1:  # random orbits around the origin
            a, p, r = rng.uniform(0, 2 * math.pi), rng.uniform(-0.35, 0.35), 0.45 * box * rng.uniform(0.8, 1.0)
            eye = (r * math.cos(p) * math.sin(a), r * math.sin(p), r * math.cos(p) * math.cos(a))
            target, fov = (0, 0, 0), 70.0
        else:  # inside the box, looking across it
            eye = np.array((0.0, 0.05, -0.45)) * box + rng.normal(0, 0.01 * box, 3)
            target, fov = rng.normal(0, 0.01 * box, 3), 70.0
        if kind in ("mixed", "batch"):
            w, h = RESOLUTIONS[v % 3 if kind == "mixed" else int(plan.integers(3))]
        out.append((slot, _f32(eye), _f32(target), fov, int(w), int(h)))
    return out


def _scenes(case, seed):
    small = case["kind"] in ("closeup", "turntable", "viewer")
    log_scale = -3.8 if case["kind"] == "closeup" else -4.0
    return [_scene(n, seed + 101 * k, not small, log_scale) for k, n in enumerate(_scene_counts(case))]


class _State:
    """What a program keeps between calls: the context, its scenes and views, the buffers it passes."""

    def __init__(self, case):
        self.case = case
        self.ctx = self.renderer = None
        self.scenes = []

    def open(self, **flags):
        c = self.case
        self.ctx = webgs.Context(tile_size=c["tile"], digit_bits=c["digit_bits"], raster_batch=c["raster_batch"],
                                 sort_block=c["sort_block"], **flags)

    def __del__(self):
        for s in self.scenes:
            s.close()
        for owner in (self.renderer, self.ctx):
            if owner is not None:
                owner.close()


def _outputs(case, width, height):
    """Device buffers of the case's outputs, by the names of Context.forward_device's arguments."""
    made = {"rgba8": lambda: torch.empty(height, width, 4, dtype=torch.uint8, device=DEV),
            "rgb": lambda: torch.empty(height, width, 3, device=DEV),
            "final_t": lambda: torch.empty(height, width, device=DEV),
            "n_contrib": lambda: torch.empty(height, width, dtype=torch.int32, device=DEV)}
    return {k: made[k]() for k in case["outputs"].split(",")}


def _image(bufs):
    p = {k: t.data_ptr() for k, t in bufs.items()}
    return _abi.Image(webgs.GS_MEM_DEVICE, p.get("rgba8"), p.get("rgb"), p.get("final_t"), p.get("n_contrib"))


def prepare(case, seed):
    s = _State(case)
    kind, w, h = case["kind"], case["width"], case["height"]
    if kind == "viewer":
        s.renderer = webgs.Renderer(w, h, tile_size=case["tile"], digit_bits=case["digit_bits"],
                                    raster_batch=case["raster_batch"], sort_block=case["sort_block"])
        s.renderer.upload_gs_data({"packed": _scenes(case, seed)[0].cpu().numpy(), "count": case["n"]}, "scene")
        s.renderer.set_gs("scene")
        s.renderer.camera.eye[:] = (0.0, 0.0, -4.0)
        s.renderer.camera.press("ShiftLeft")  # the mouse turns the camera while shift is held
        s.turn = 3.0
        return s
    training = kind in ("train", "train_batch")
    s.open(flags=webgs.GS_FLAG_DIFFERENTIABLE if training else 0)
    if kind == "loss":
        s.x, s.y = _photo(w, h, seed), _photo(w, h, seed + 1)
        s.x = (0.9 * s.y + 0.1 * s.x).contiguous()  # a render near its target
        s.dl = torch.empty(h, w, 3, device=DEV)
        torch.cuda.synchronize()
        return s
    packed = _scenes(case, seed)
    cams = _cameras(case, seed)
    torch.cuda.synchronize()  # the context's stream is its own: the scene is there before it reads it
    s.scenes = [s.ctx.upload(p.data_ptr(), n, webgs.GS_MEM_DEVICE) for p, n in zip(packed, _scene_counts(case))]
    s.views = [webgs.camera_view(eye, target, (0.0, 1.0, 0.0), fov, cw, ch, NEAR, FAR)
               for _, eye, target, fov, cw, ch in cams]
    if training:
        s.packed = packed[0]
        s.target = [_photo(w, h, seed + 13 * k) for k in range(len(cams))]
        s.rgb = [torch.empty(h, w, 3, device=DEV) for _ in cams]
        s.dl = [torch.empty(h, w, 3, device=DEV) for _ in cams]
        s.grad = torch.empty(59 * case["n"], device=DEV)
        s.dl_ptrs = (C.c_void_p * len(cams))(*[t.data_ptr() for t in s.dl])
        s.out = [{"rgb": t} for t in s.rgb]
    else:
        s.out = [_outputs(case, cw, ch) for *_, cw, ch in cams]
    if kind in ("batch", "train_batch"):
        s.items = (_abi.BatchView * len(cams))()
        for i, (slot, *_) in enumerate(cams):
            s.items[i].scene, s.items[i].view, s.items[i].out = s.scenes[slot].handle, s.views[i], _image(s.out[i])
    elif kind == "turntable":
        s.items = (_abi.BatchCamera * len(cams))()
        for i, (slot, eye, target, fov, cw, ch) in enumerate(cams):
            cam = webgs.make_camera(eye, target, (0.0, 1.0, 0.0), fov, cw, ch, NEAR, FAR)
            s.items[i].scene, s.items[i].camera, s.items[i].out = s.scenes[slot].handle, cam, _image(s.out[i])
    torch.cuda.synchronize()
    return s


# ---- one pass --------------------------------------------------------------------------------------
def _ok(s, rc):
    if rc != _abi.GS_OK:
        raise webgs.GsError(rc, webgs.library().gs_last_error(s.ctx.handle).decode())


def _loss(s, k, value):
    h, w = s.rgb[k].shape[:2]
    _ok(s, webgs.library().gs_loss_l1_ssim(s.ctx.handle, s.rgb[k].data_ptr(), s.target[k].data_ptr(), w, h, LAMBDA,
                                           value, s.dl[k].data_ptr(), webgs.GS_MEM_DEVICE))


def run(state):
    s, kind, lib = state, state.case["kind"], webgs.library()
    if kind == "viewer":
        s.turn = -s.turn
        s.renderer.camera.mouse_move(s.turn, 0.0)
        s.renderer.execute(1.0 / 60.0)
        return s.renderer.image
    if kind == "loss":
        h, w = s.x.shape[:2]
        value = C.c_double()
        _ok(s, lib.gs_loss_l1_ssim(s.ctx.handle, s.x.data_ptr(), s.y.data_ptr(), w, h, LAMBDA, C.byref(value),
                                   s.dl.data_ptr(), webgs.GS_MEM_DEVICE))
        return {"loss": value.value, "dl": s.dl}
    if kind in ("frame", "closeup", "mixed"):
        for view, bufs in zip(s.views, s.out):
            s.ctx.forward_device(s.scenes[0], view, **{k: t.data_ptr() for k, t in bufs.items()})
        return s.out
    if kind == "batch":
        _ok(s, lib.gs_forward_batch(s.ctx.handle, s.items, len(s.items)))
        return s.out
    if kind == "turntable":
        _ok(s, lib.gs_forward_batch_cameras(s.ctx.handle, s.items, len(s.items)))
        return s.out
    # a training step: the optimizer's attributes, then forward, loss and backward
    s.scenes[0].update(s.packed.data_ptr(), webgs.GS_MEM_DEVICE)
    if kind == "train":
        value = C.c_double()
        s.ctx.forward_device(s.scenes[0], s.views[0], rgb=s.rgb[0].data_ptr())
        _loss(s, 0, C.byref(value))
        _ok(s, lib.gs_backward(s.ctx.handle, s.scenes[0].handle, s.dl[0].data_ptr(), s.grad.data_ptr(),
                               webgs.GS_MEM_DEVICE))
        return {"loss": value.value, "rgb": s.rgb[0], "grad": s.grad}
    _ok(s, lib.gs_forward_batch(s.ctx.handle, s.items, len(s.items)))
    for k in range(len(s.rgb)):
        _loss(s, k, None)
    _ok(s, lib.gs_backward_batch(s.ctx.handle, s.scenes[0].handle, s.dl_ptrs, len(s.dl), s.grad.data_ptr(),
                                 webgs.GS_MEM_DEVICE))
    return {"rgb": s.rgb, "grad": s.grad}


def work(case):
    """Bytes: attributes read once, images and gradients moved once. Flops: about 700 per Gaussian and
    view for the projection and the SH, 65 blended splats per pixel (the scenes' mean) of 45 operations,
    three times that with the backward, and 440 per pixel and channel for the loss's filters."""
    kind, views = case["kind"], case["views"]
    sizes = [(case["width"], case["height"])] * views
    if kind in ("mixed", "batch"):
        sizes = [RESOLUTIONS[v % 3] for v in range(views)]
    pixels = sum(w * h for w, h in sizes)
    if kind == "loss":
        return {"bytes": 36.0 * pixels, "flops": 3 * 440.0 * pixels}
    n = sum(_scene_counts(case))
    if kind in ("train", "train_batch"):
        return {"bytes": 2 * 236.0 * n + 24.0 * pixels,
                "flops": 2100.0 * n * views + (3 * 65 * 45.0 + 3 * 440.0) * pixels}
    per_pixel = {"rgba8": 4, "rgb": 12, "final_t": 4, "n_contrib": 4}
    out = sum(per_pixel[k] for k in case["outputs"].split(","))
    return {"bytes": 236.0 * n + out * pixels, "flops": 700.0 * n * views / (3 if kind == "batch" else 1) + 65 * 45.0 * pixels}


# ---- the same in 64 bits ---------------------------------------------------------------------------
def _uniforms(eye, target, fov, width, height):
    """The view's float32 uniforms (the pipeline's input) in float64: view and view-projection matrices
    (row, column), focal lengths and tangents."""
    e, t, up = (np.array(v, np.float64) for v in (eye, target, (0.0, 1.0, 0.0)))
    unit = lambda v: v / np.linalg.norm(v)  # noqa: E731
    z = unit(e - t)
    x = unit(np.cross(up, z))
    y = unit(np.cross(z, x))
    view = np.eye(4)
    for r, axis in enumerate((x, y, z)):
        view[r, :3], view[r, 3] = axis, -axis @ e
    view = view.astype(np.float32).astype(np.float64)
    aspect, fovy = width / height, math.radians(fov)
    f = 1.0 / math.tan(fovy / 2)
    proj = np.zeros((4, 4))
    proj[0, 0], proj[1, 1], proj[3, 2] = f / aspect, f, -1.0
    near, far = float(np.float32(NEAR)), float(np.float32(FAR))
    proj[2, 2], proj[2, 3] = far / (near - far), far * near / (near - far)
    proj = proj.astype(np.float32).astype(np.float64)
    tan_y = math.tan(fovy / 2)
    small = np.array([width / (2 * tan_y * aspect), height / (2 * tan_y), tan_y * aspect, tan_y], np.float32)
    as64 = lambda m: torch.tensor(np.asarray(m, np.float32).astype(np.float64), device=DEV)  # noqa: E731
    return {"view": as64(view), "view_proj": as64(proj @ view), "eye": as64(e), "focal": small[:2].astype(float),
            "tan": small[2:].astype(float)}


def _project(packed, u, width, height, tile):
    """Each Gaussian's pixel position, conic, opacity and colour (differentiable), its tile rectangle and
    16-bit depth; culled Gaussians have no tiles."""
    n = packed.numel() // 59
    pos, scale, quat, dc, logit, rest = torch.split(packed, [3 * n, 3 * n, 4 * n, 3 * n, n, 45 * n])
    pos, scale, quat, dc, rest = pos.view(n, 3), scale.view(n, 3), quat.view(n, 4), dc.view(n, 3), rest.view(n, 3, 15)
    one = torch.ones(n, 1, dtype=torch.float64, device=DEV)
    hom = torch.cat([pos, one], 1)
    pv, clip = hom @ u["view"].T, hom @ u["view_proj"].T
    near = pv[:, 2].detach() < -0.2
    ndc = clip[:, :3] / (clip[:, 3:] + 1e-7)
    size = torch.tensor([width, height], dtype=torch.float64, device=DEV)
    pix = ((ndc[:, :2] + 1) * size - 1) * 0.5
    w, x, y, z = (quat / quat.norm(dim=1, keepdim=True)).unbind(1)
    rot = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                       2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                       2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).view(n, 3, 3)
    a = rot * scale.exp()[:, None, :]
    tz = pv[:, 2]
    t = []
    for k in range(2):  # outside the guard band the clamped coordinate passes no gradient
        lim = 1.3 * u["tan"][k]
        ratio = (pv[:, k] / tz).detach()
        t.append(torch.where(ratio.abs() > lim, ratio.clamp(-lim, lim) * tz.detach(), pv[:, k]))
    zero = torch.zeros_like(tz)
    fx, fy = u["focal"]
    jac = torch.stack([fx / tz, zero, -fx * t[0] / (tz * tz), zero, fy / tz, -fy * t[1] / (tz * tz)], 1).view(n, 2, 3)
    half = (jac @ u["view"][:3, :3]) @ a
    cov = half @ half.transpose(1, 2)
    ca, cb, cc = cov[:, 0, 0] + 0.3, cov[:, 0, 1], cov[:, 1, 1] + 0.3
    det = ca * cc - cb * cb
    conic = torch.stack([cc / det, -cb / det, ca / det], 1)
    d = pos - u["eye"]
    x, y, z = (d / d.norm(dim=1, keepdim=True)).unbind(1)
    xx, yy, zz = x * x, y * y, z * z
    c2, c3 = 1.0925484305920792, 0.5900435899266435
    basis = torch.stack([-0.4886025119029199 * y, 0.4886025119029199 * z, -0.4886025119029199 * x, c2 * x * y,
                         -c2 * y * z, 0.31539156525252005 * (2 * zz - xx - yy), -c2 * x * z, 0.5462742152960396 * (xx - yy),
                         -c3 * y * (3 * xx - yy), 2.890611442640554 * x * y * z, -0.4570457994644658 * y * (4 * zz - xx - yy),
                         0.3731763325901154 * z * (2 * zz - 3 * xx - 3 * yy), -0.4570457994644658 * x * (4 * zz - xx - yy),
                         1.445305721320277 * z * (xx - yy), -c3 * x * (xx - 3 * yy)], 1)
    colour = (0.28209479177387814 * dc + (rest * basis[:, None, :]).sum(2) + 0.5).clamp_min(0)
    with torch.no_grad():
        mid = 0.5 * (ca + cc)
        radius = (3 * (mid + (mid * mid - det).clamp_min(0.1).sqrt()).sqrt()).ceil()
        lo, hi = pix - radius[:, None], pix + radius[:, None]
        seen = near & (hi >= 0).all(1) & (lo <= size).all(1)
        tiles = torch.tensor([-(-width // tile), -(-height // tile)], device=DEV)
        lo, hi = (torch.minimum((v / tile).floor().clamp_min(0), (tiles - 1).double()).nan_to_num().long() for v in (lo, hi))
        count = torch.where(seen, (hi - lo + 1).prod(1), 0)
        depth = (ndc[:, 2].clamp(0, 1) * 65535).nan_to_num().long()
    return pix, conic, torch.sigmoid(logit), colour, (lo, hi, count, depth)


def _instances(rect, width, tile):
    """Gaussian of every (tile, splat) pair in drawing order, and each tile's part of that list."""
    lo, hi, count, depth = rect
    g = torch.repeat_interleave(torch.arange(count.numel(), device=DEV), count)
    k = torch.arange(g.numel(), device=DEV) - (count.cumsum(0) - count)[g]
    span = (hi - lo + 1)[g, 0]
    at = (lo[g, 1] + k // span) * (-(-width // tile)) + lo[g, 0] + k % span
    key, order = torch.sort(at * 65536 + depth[g], stable=True)
    return g[order], key // 65536


class _Raster64:
    """Front-to-back blending of every tile at once, one range position after the other, and its adjoint."""
    STEP = 64  # positions between two looks at which tiles are still at work

    def __init__(self, pix, conic, opacity, colour, rect, width, height, tile):
        self.par = torch.cat([pix, conic, opacity[:, None], colour], 1).detach()
        self.vals, tiles = _instances(rect, width, tile)
        tx, ty = -(-width // tile), -(-height // tile)
        self.lens = torch.bincount(tiles, minlength=tx * ty)
        self.starts = self.lens.cumsum(0) - self.lens
        at, px = torch.arange(tx * ty, device=DEV), torch.arange(tile * tile, device=DEV)
        self.x = ((at % tx) * tile)[:, None] + px % tile
        self.y = ((at // tx) * tile)[:, None] + px // tile
        self.inside = (self.x < width) & (self.y < height)
        self.width, self.height = width, height
        self.T = torch.ones(self.x.shape, dtype=torch.float64, device=DEV)
        self.C = torch.zeros(*self.x.shape, 3, dtype=torch.float64, device=DEV)
        self.last = torch.zeros_like(self.x)

    def _eval(self, sel, r, fx, fy):
        valid = r < self.lens[sel]
        g = self.vals[(self.starts[sel] + r).clamp_max(max(self.vals.numel() - 1, 0))]
        q = self.par[g]
        dx, dy = q[:, 0, None] - fx, q[:, 1, None] - fy
        power = -0.5 * (q[:, 2, None] * dx * dx + q[:, 4, None] * dy * dy) - q[:, 3, None] * dx * dy
        e = power.exp()
        raw = q[:, 5, None] * e
        alpha = raw.clamp_max(0.99)
        return g, q, dx, dy, e, raw, alpha, valid[:, None] & (power <= 0) & (alpha >= 1.0 / 255.0)

    def forward(self):
        done = ~self.inside
        r0 = 0
        while True:
            sel = ((self.lens > r0) & ~done.all(1)).nonzero()[:, 0]
            if not sel.numel():
                break
            fx, fy = self.x[sel].double(), self.y[sel].double()
            T, col, dn, last = self.T[sel], self.C[sel], done[sel], self.last[sel]
            for r in range(r0, r0 + self.STEP):
                _, q, _, _, _, _, alpha, hit = self._eval(sel, r, fx, fy)
                hit &= ~dn
                test = T * (1 - alpha)
                stop = hit & (test < 1e-4)
                hit &= ~stop
                dn |= stop
                w = torch.where(hit, alpha * T, 0.0)
                col += w[..., None] * q[:, None, 6:9]
                T = torch.where(hit, test, T)
                last = torch.where(hit, r + 1, last)
            self.T[sel], self.C[sel], done[sel], self.last[sel] = T, col, dn, last
            r0 += self.STEP
        return self._to_image(self.C), self._to_image(self.T[..., None])[..., 0]

    def _to_image(self, v):
        img = torch.zeros(self.height, self.width, v.shape[-1], dtype=torch.float64, device=DEV)
        img[self.y[self.inside], self.x[self.inside]] = v[self.inside]
        return img

    def backward(self, dl):
        """Gradient of each Gaussian's nine raster parameters."""
        grad = torch.zeros_like(self.par)
        d_all = dl[self.y.clamp_max(self.height - 1), self.x.clamp_max(self.width - 1)] * self.inside[..., None]
        T_all, S_all = self.T.clone(), torch.zeros_like(self.T)  # S: dL/dC . colour added behind the splat
        top = self.last.amax(1)
        for r0 in range((max(int(top.max()) - 1, 0) // self.STEP) * self.STEP, -1, -self.STEP):
            sel = (top > r0).nonzero()[:, 0]
            if not sel.numel():
                continue
            fx, fy = self.x[sel].double(), self.y[sel].double()
            T, S, last, d = T_all[sel], S_all[sel], self.last[sel], d_all[sel]
            for r in range(r0 + self.STEP - 1, r0 - 1, -1):
                g, q, dx, dy, e, raw, alpha, hit = self._eval(sel, r, fx, fy)
                hit &= r < last
                T = torch.where(hit, T / (1 - alpha), T)
                w = torch.where(hit, alpha * T, 0.0)
                k = (d * q[:, None, 6:9]).sum(2)
                da = torch.where(hit & (raw <= 0.99), T * k - S / (1 - alpha), 0.0)
                gp = da * raw
                a, b, c = q[:, 2, None], q[:, 3, None], q[:, 4, None]
                parts = [-(gp * (a * dx + b * dy)).sum(1), -(gp * (b * dx + c * dy)).sum(1), -0.5 * (gp * dx * dx).sum(1),
                         -(gp * dx * dy).sum(1), -0.5 * (gp * dy * dy).sum(1), (da * e).nan_to_num(posinf=0.0).sum(1)]
                grad.index_add_(0, g, torch.cat([torch.stack(parts, 1), (w[..., None] * d).sum(1)], 1))
                S = S + w * k
            T_all[sel], S_all[sel] = T, S
        return grad


def _loss64(x, y):
    """L1 + lambda (1 - SSIM) and dL/dx: 11x11 Gaussian window, sigma 1.5, zero padding."""
    x = x.detach().clone().requires_grad_(True)
    k = torch.exp(-((torch.arange(11, dtype=torch.float64, device=DEV) - 5) ** 2) / 4.5)
    k = k / k.sum()

    def blur(v):
        for axis in (0, 1):
            size = v.shape[axis]
            v = torch.nn.functional.pad(v, (0, 0) + (0, 0) * (1 - axis) + (5, 5))
            v = sum(k[i] * v.narrow(axis, i, size) for i in range(11))
        return v

    mx, my = blur(x), blur(y)
    sxx, syy, sxy = blur(x * x) - mx * mx, blur(y * y) - my * my, blur(x * y) - mx * my
    c1, c2 = 0.01 ** 2, 0.03 ** 2
    ssim = ((2 * mx * my + c1) * (2 * sxy + c2)) / ((mx * mx + my * my + c1) * (sxx + syy + c2))
    loss = (x - y).abs().mean() + LAMBDA * (1 - ssim.mean())
    loss.backward()
    return float(loss.detach()), x.grad


def exact(case, seed):
    kind, w, h = case["kind"], case["width"], case["height"]
    if kind == "loss":
        y = _photo(w, h, seed + 1)
        x = (0.9 * y + 0.1 * _photo(w, h, seed)).contiguous()
        loss, dl = _loss64(x.double(), y.double())
        return {"loss": loss, "dl": dl}
    asked = case["outputs"].split(",")
    training = kind in ("train", "train_batch")
    if kind in ("viewer", "turntable", "batch") or not (training or {"rgb", "final_t"} & set(asked)):
        return None  # bytes and counts only
    packed = _scenes(case, seed)[0].double().requires_grad_(training)
    grad, out = torch.zeros_like(packed), []
    loss = None
    for k, (_, eye, target, fov, cw, ch) in enumerate(_cameras(case, seed)):
        u = _uniforms(eye, target, fov, cw, ch)
        with torch.set_grad_enabled(training):
            *par, rect = _project(packed, u, cw, ch, case["tile"])
        with torch.no_grad():
            raster = _Raster64(*par, rect, cw, ch, case["tile"])
            rgb, final_t = raster.forward()
        if not training:
            found = {"rgb": rgb, "final_t": final_t}
            out.append({name: found.get(name) for name in asked})
            continue
        loss, dl = _loss64(rgb, _photo(cw, ch, seed + 13 * k).double())
        with torch.no_grad():
            g2 = raster.backward(dl)
        near = rect[2] > 0  # culled Gaussians get no gradient
        flat = torch.cat([par[0], par[1], par[2][:, None], par[3]], 1)
        total = (flat[near] * g2[near]).sum()
        grad += torch.autograd.grad(total, packed)[0].nan_to_num(0.0)
        out.append(rgb)
        del raster, par, rect, flat, total
    if kind == "train":
        return {"loss": loss, "rgb": out[0], "grad": grad}
    if kind == "train_batch":
        return {"rgb": out, "grad": grad}
    return out
