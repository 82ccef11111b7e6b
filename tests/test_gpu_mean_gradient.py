"""The screen-mean gradient of elongated, tilted Gaussians (src/rasterize.rs:434-451), where the
terms A dx and B dy of a pixel nearly cancel: the default backward's error against 64 bits is no
larger than that of the deterministic one, which sums every pixel's term as the reference does.

One Gaussian per tile, so that its gradient is a plain sum over the tile's pixels. The 64-bit sum
takes sigma and the pixels' decisions in float32, operation for operation as every backward does;
what is compared is the sum's own rounding. Both roundings of a pixel's A dx + B dy dominate the
deterministic error; the default backward has one of them (a fused multiply-add), hence 0.7 of
that error, and a bound of 1."""
import numpy as np
import pytest
import torch

from splatrs_b200 import gpu as G

pytestmark = pytest.mark.gpu

EDGE = 64  # tiles per side
SIZE = (16 * EDGE, 16 * EDGE)
OPACITY = np.float32(0.6)


def tilted(major, minor, seed):
    """One reference projection record per tile: axes in pixels, any angle."""
    rng = np.random.default_rng(seed)
    ty, tx = np.divmod(np.arange(EDGE * EDGE), EDGE)
    p = np.zeros((EDGE * EDGE, 15), np.float32)
    p[:, 0] = 16 * tx + rng.uniform(5.0, 11.0, tx.size)
    p[:, 1] = 16 * ty + rng.uniform(5.0, 11.0, tx.size)
    angle = rng.uniform(0.0, np.pi, tx.size)
    c, s, l1, l2 = np.cos(angle), np.sin(angle), major ** -2.0, minor ** -2.0
    p[:, 2], p[:, 4] = l1 * c * c + l2 * s * s, l1 * s * s + l2 * c * c
    p[:, 3] = (l1 - l2) * c * s
    p[:, 5], p[:, 6], p[:, 7] = 1.0, 20.0, OPACITY
    p[:, 8:11] = 1.0
    p[:, 11], p[:, 12], p[:, 13], p[:, 14] = tx, ty, tx + 1, ty + 1
    return p


def exact(p, dimage):
    """(gradient of the mean, sum of the terms' magnitudes), (n, 2) each, in 64 bits."""
    n = len(p)
    tiles = dimage.reshape(EDGE, 16, EDGE, 16, 3).transpose(0, 2, 1, 3, 4).reshape(n, 16, 16, 3)
    x = np.float32(16.0) * p[:, 11, None, None] + np.arange(16, dtype=np.float32)[None, None, :] + np.float32(0.5)
    y = np.float32(16.0) * p[:, 12, None, None] + np.arange(16, dtype=np.float32)[None, :, None] + np.float32(0.5)
    mx, my, a, b, c = (p[:, k, None, None] for k in range(5))
    dx, dy = x - mx, y - my
    sigma = np.float32(0.5) * (a * dx * dx + c * dy * dy) + b * dx * dy
    with np.errstate(over="ignore"):
        gauss = np.exp(-sigma.astype(np.float64))
    alpha = OPACITY * gauss.astype(np.float32)
    taken = (sigma >= 0) & (alpha >= np.float32(1.0) / np.float32(255.0))
    # A lone entry: T = 1, no colour behind it and a black background.
    h = np.where(taken, gauss, 0.0) * tiles.astype(np.float64).sum(3) * np.float64(OPACITY)
    a, b, c, dx, dy = (v.astype(np.float64) for v in (a, b, c, dx, dy))
    terms = np.stack([h * (a * dx + b * dy), h * (b * dx + c * dy)], 3)
    return terms.sum((1, 2)), np.abs(terms).sum((1, 2))


@pytest.mark.parametrize("major,minor", [(10.0, 0.2), (50.0, 0.1), (200.0, 0.1)])
def test_mean_gradient_of_elongated_gaussians(major, minor):
    p = tilted(major, minor, int(major))
    dimage = np.random.default_rng(7).normal(0, 1, SIZE[0] * SIZE[1] * 3).astype(np.float32)
    want, scale = exact(p, dimage)
    ctx = G.Context(0)
    black = np.zeros(3, np.float32)
    proj = G.proj_from_reference(ctx, torch.from_numpy(p).cuda(), *SIZE)
    b = G.bin(ctx, proj)
    out = G.rasterize_forward(ctx, proj, b, black)
    d = torch.from_numpy(dimage).cuda()
    got = [G.pgrad_to_reference(f(ctx, proj, b, black, out, d), len(p))[0].cpu().numpy()[:, :2].astype(np.float64)
           for f in (G.rasterize_backward, G.rasterize_backward_deterministic)]
    ctx.close()
    live = (scale > 0).all(1)
    assert live.mean() > 0.9
    rms = [np.sqrt((((g - want) / np.maximum(scale, 1e-30))[live] ** 2).mean(0)) for g in got]
    print(f"\naxes {major} and {minor}: error / sum of magnitudes, default {rms[0]}, deterministic {rms[1]}")
    assert (rms[1] < 1e-5).all()  # the 64-bit sum is of the same pixels
    assert (rms[0] <= rms[1]).all()
