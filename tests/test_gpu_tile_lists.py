"""Compositing over tile lists whose lengths sit at the edges of the warps' walk: 32-entry stages
(16 in the backward), the 1,024-entry scan, lists that pixels leave early, and entries that
take the scalar rule (opacity above 1, a conic beyond the plain range). Projections are made
here and handed to the device and to the oracle (src/rasterize.rs:249-505) alike."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from splatrs_b200 import gpu as G

pytestmark = pytest.mark.gpu

SIZE = (27, 22)  # 2 x 2 tiles of 16, ragged on both sides
BG = np.array((0.3, 0.6, 0.1), np.float32)


@pytest.fixture(scope="module")
def ctx():
    c = G.Context(0)
    yield c
    c.close()


@pytest.fixture
def cr_math():
    O.set_cr_math(True)
    yield
    O.set_cr_math(False)


def projections(n, opacity, seed, special=False):
    """n reference projection records covering every tile of the image."""
    rng = np.random.default_rng(seed)
    p = np.zeros((n, 15), np.float32)
    p[:, 0] = rng.uniform(-4.0, SIZE[0] + 4.0, n)
    p[:, 1] = rng.uniform(-4.0, SIZE[1] + 4.0, n)
    a, c = rng.uniform(0.02, 1.5, n), rng.uniform(0.02, 1.5, n)
    p[:, 2], p[:, 4] = a, c
    p[:, 3] = rng.uniform(-0.8, 0.8, n) * np.sqrt(a * c)
    p[:, 5] = rng.uniform(1.0, 9.0, n)
    p[:, 6] = 12
    p[:, 7] = rng.uniform(0.6, 1.4, n) * opacity
    p[:, 8:11] = rng.uniform(0.0, 1.0, (n, 3))
    p[:, 13:15] = 2
    if special:
        p[::3, 7] = 2.0     # ln(255 opacity) above the table's range; alpha clamps
        p[1::7, 2:5] = (1e16, 0.0, 1e16)
    return p


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


# Gradients: every quantity within 1e-3 of its scale, the bar of the other backward tests.
@pytest.mark.parametrize("tile", [(16, 16), (8, 8), (16, 32)])
@pytest.mark.parametrize("n,opacity,special", [
    (1, 0.5, False), (7, 0.5, False), (9, 0.5, True), (16, 0.2, False), (17, 0.2, False), (31, 0.1, False),
    (32, 0.1, False), (33, 0.1, True), (65, 0.05, False), (1024, 0.01, False), (1025, 0.01, False),
    (2100, 0.01, True), (1500, 0.6, False)])
def test_lists_at_the_edges_of_a_walk(ctx, cr_math, tile, n, opacity, special):
    p = projections(n, opacity, 100 + n, special)
    dimage = np.random.default_rng(n).normal(0, 1, SIZE[0] * SIZE[1] * 3).astype(np.float32)
    ob = O.bin(p, *SIZE)
    img, ft, nc, pairs = O.rasterize_forward(p, ob, *SIZE, BG)
    og, oa, opairs = O.rasterize_backward(p, ob, *SIZE, BG, ft, nc, dimage)
    ctx.raster_config = (*tile, 256, 2)
    try:
        proj = G.proj_from_reference(ctx, dev(p), *SIZE)
        b = G.bin(ctx, proj)
        out = G.rasterize_forward(ctx, proj, b, BG)
        got_pairs = torch.zeros(1, dtype=torch.int64, device="cuda")
        pg = G.rasterize_backward(ctx, proj, b, BG, out, dev(dimage), pairs=got_pairs)
        plain = G.rasterize_backward(ctx, proj, b, BG, out, dev(dimage))
    finally:
        ctx.raster_config = (16, 16, 256, 2)
    assert (bits(out.image.cpu().numpy()) == bits(img)).all()
    assert (bits(out.final_t.cpu().numpy()) == bits(ft)).all()
    if tile == (16, 16):
        assert (out.n_contrib.cpu().numpy().view(np.uint32) == nc).all()
    assert int(out.pairs.item()) == pairs and int(got_pairs.item()) == opairs
    for pgrad in (pg, plain):
        gg, ga = (v.cpu().numpy() for v in G.pgrad_to_reference(pgrad, n))
        for got, want in ((gg, og), (ga, oa)):
            scale = np.maximum(np.abs(want).max(0), 1e-30)
            assert (np.abs(got - want).max(0) / scale).max() < 1e-3


@pytest.mark.parametrize("tile", [(16, 16), (8, 8), (16, 32)])
@pytest.mark.parametrize("n", [40, 1100, 2300])
def test_warps_that_saturate_early(ctx, cr_math, tile, n):
    """Opaque entries in front close the pixels around one corner of a tile, while those of the
    other corners go through the whole list, over one, two and three scans of it: the backward's
    warps start at places of their own."""
    p = projections(n, 0.4 / np.sqrt(n), 500 + n)
    p[:12, :5] = (4.0, 4.0, 0.02, 0.0, 0.02)
    p[:12, 5], p[:12, 6], p[:12, 7] = 0.5 + 0.01 * np.arange(12), 3.0, 0.99
    dimage = np.random.default_rng(n).normal(0, 1, SIZE[0] * SIZE[1] * 3).astype(np.float32)
    ob = O.bin(p, *SIZE)
    img, ft, nc, _ = O.rasterize_forward(p, ob, *SIZE, BG)
    og, oa, opairs = O.rasterize_backward(p, ob, *SIZE, BG, ft, nc, dimage)
    assert nc.min() <= 8 and nc.max() > 0.9 * n
    ctx.raster_config = (*tile, 256, 2)
    try:
        proj = G.proj_from_reference(ctx, dev(p), *SIZE)
        b = G.bin(ctx, proj)
        out = G.rasterize_forward(ctx, proj, b, BG)
        got_pairs = torch.zeros(1, dtype=torch.int64, device="cuda")
        pgrad = G.rasterize_backward(ctx, proj, b, BG, out, dev(dimage), pairs=got_pairs)
    finally:
        ctx.raster_config = (16, 16, 256, 2)
    assert (bits(out.image.cpu().numpy()) == bits(img)).all()
    assert int(got_pairs.item()) == opairs
    for got, want in zip((v.cpu().numpy() for v in G.pgrad_to_reference(pgrad, n)), (og, oa)):
        scale = np.maximum(np.abs(want).max(0), 1e-30)
        assert (np.abs(got - want).max(0) / scale).max() < 1e-3
