"""The raster backward's sums over a block of 8x4 pixels, by themselves: small splats far apart, each near a corner
of a block, under a dL/drgb of one sign, so that no other splat and no recovered transmittance takes part.
Their gradients with respect to colour, opacity and the scales across the view follow in 64 bits from the
projected values that the frame gives (pixel, conic, opacity): sums over pixels of gp, gp dx^2, gp dx dy, gp dy^2
and w dC, which are formed about the splat's centre. Once with dL/drgb at the corner pixels alone (a pixel to a
splat, 0.1 to 0.45 pixels from its centre), where sums formed about anything else would cancel, and once everywhere.

Tolerance: nothing here cancels, so a gradient carries the roundings it went through one after the other, at
most 64 of 2^-24 each from the exp to the packed attribute: 4e-6 of the gradient."""
import numpy as np
import pytest

import webgs
from webgs import workloads as W

pytestmark = pytest.mark.gpu
TOL = 64 * 2.0 ** -24
SH_C0 = 0.28209479177387814


def _splats(ctx, view, w, h):
    """One splat per 24x12 pixels near a corner of an 8x4 block, facing the camera: (packed, corner pixels)."""
    probe = np.zeros(59 * 3, np.float32)
    probe[:9] = (0, 0, 0, 1, 0, 0, 0, 1, 0)
    probe[9:18] = -4.0
    probe[18:30] = (1, 0, 0, 0) * 3
    sc = ctx.upload(probe, 3)
    ctx.forward(sc, view)
    p = ctx.debug()["pixel"].reshape(3, 2).astype(np.float64)
    sc.close()
    rng = np.random.default_rng(11)
    bx, by = [v.ravel() for v in np.meshgrid(np.arange(1, w // 8 - 1, 3), np.arange(2, h // 4 - 2, 3))]
    n = len(bx)
    right, below = rng.integers(0, 2, n), rng.integers(0, 2, n)
    corner = np.stack([8 * bx + 7 * right, 4 * by + 3 * below], 1)
    at = corner + rng.uniform(0.1, 0.45, (n, 2)) * rng.choice([-1.0, 1.0], (n, 2))
    pos = np.zeros((n, 3))
    pos[:, :2] = np.linalg.solve(np.stack([p[1] - p[0], p[2] - p[0]], 1), (at - p[0]).T).T
    packed = np.zeros(59 * n, np.float32)
    packed[:3 * n] = pos.ravel()
    packed[3 * n:6 * n] = np.log(0.3 * 4.0 / view.focal[0])  # 0.3 pixels before the low-pass
    packed[6 * n:10 * n] = np.tile((1, 0, 0, 0), n)
    packed[10 * n:13 * n] = rng.uniform(0.2, 2.0, 3 * n)
    packed[13 * n:14 * n] = rng.uniform(-3.0, 0.0, n)
    return packed, corner


@pytest.mark.parametrize("tile", [8, 16, 32])
@pytest.mark.parametrize("where", ["corners", "everywhere"])
def test_sums_over_a_block(where, tile):
    w, h = 256, 160
    view = W.CameraSpec((0.0, 0.0, -4.0), (0.0, 0.0, 0.0), 60.0, w, h).view()
    with webgs.Context(flags=webgs.GS_FLAG_DIFFERENTIABLE, tile_size=tile) as ctx:
        packed, corner = _splats(ctx, view, w, h)
        n = len(corner)
        dl = np.random.default_rng(12).uniform(0.5e-3, 1.5e-3, (h, w, 3)).astype(np.float32)
        if where == "corners":
            on = np.zeros((h, w, 1), bool)
            on[corner[:, 1], corner[:, 0]] = True
            dl = np.where(on, dl, 0.0).astype(np.float32)
        sc = ctx.upload(packed, n)
        ctx.forward(sc, view, rgba8=False, rgb=True)
        dbg = ctx.debug()
        got = ctx.backward(sc, dl).astype(np.float64)
        sc.close()
    centre = dbg["pixel"].reshape(n, 2).astype(np.float64)
    conic = dbg["conic_opacity"].reshape(n, 4).astype(np.float64)
    colour = dbg["color"].reshape(n, 4)[:, :3].astype(np.float64)
    want_scale, want_dc, want_op = np.zeros((n, 2)), np.zeros((n, 3)), np.zeros(n)
    for g in range(n):
        A, B, C, o = conic[g]
        x, y = np.meshgrid(np.arange(corner[g, 0] - 8, corner[g, 0] + 9), np.arange(corner[g, 1] - 6, corner[g, 1] + 7))
        dx, dy = centre[g, 0] - x, centre[g, 1] - y
        alpha = o * np.exp(-0.5 * (A * dx * dx + C * dy * dy) - B * dx * dy)
        assert np.abs(alpha * 255.0 - 1.0).min() > 1e-5  # no pixel whose decision 32 bits could turn
        d = np.where((alpha * 255.0 >= 1.0)[..., None], dl[y, x].astype(np.float64), 0.0)
        gp = alpha * (d @ colour[g])
        want_dc[g] = SH_C0 * (alpha[..., None] * d).sum((0, 1))
        want_op[g] = gp.sum() * (1.0 - o)
        m = np.array([[A, B], [B, C]])
        grad = np.array([[-0.5 * (gp * dx * dx).sum(), -0.5 * (gp * dx * dy).sum()],
                         [-0.5 * (gp * dx * dy).sum(), -0.5 * (gp * dy * dy).sum()]])
        cov = -m @ grad @ m
        depth = 4.0
        s2 = np.exp(2.0 * packed[3 * n + 3 * g:3 * n + 3 * g + 2].astype(np.float64))
        want_scale[g] = 2.0 * s2 * (np.array([view.focal[0], view.focal[1]], np.float64) / depth) ** 2 * np.diag(cov)
    assert want_op.min() > 0.0
    for name, a, b in (("scale", got[3 * n:6 * n].reshape(n, 3)[:, :2], want_scale),
                       ("dc", got[10 * n:13 * n].reshape(n, 3), want_dc), ("opacity", got[13 * n:14 * n], want_op)):
        err = np.abs(a / b - 1.0).max()
        print(name, err)
        assert err <= TOL, (name, err)
