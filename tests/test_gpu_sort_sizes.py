"""The binning sort (src/rasterize.rs:76-119) at the edges of its tile shapes, and with keys that
do not fit the Gaussian beside tile and depth in 64 bits: every entry's Gaussian, the reference
keys and the tile ranges against a stable numpy sort, host- and device-driven."""
import numpy as np
import pytest
import torch

from splatrs_b200 import gpu as G

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = G.Context(0)
    yield c
    c.close()


# (entries, image size, smallest and largest depth): one tile per Gaussian.
@pytest.mark.parametrize("n,size,lo,hi", [
    (1, (640, 480), 1.0, 1.0), (2, (16, 16), 1.0, 2.0), (1024, (640, 480), 0.5, 9.0), (1025, (640, 480), 0.5, 9.0),
    (4097, (33, 17), 0.5, 9.0), (65536, (640, 480), 0.5, 9.0), (65537, (640, 480), 0.5, 9.0),
    (786432, (1920, 1080), 0.5, 9.0), (786433, (1920, 1080), 0.5, 9.0), (1100003, (1920, 1080), 3.0, 3.5),
    (140001, (4096, 4096), 1e-30, 1e30)])  # 16 + 31 + 18 bits: the Gaussian travels beside the key
def test_sort_at_the_edges_of_its_shapes(ctx, n, size, lo, hi):
    rng = np.random.default_rng(n)
    tiles_x, tiles_y = (size[0] + 15) // 16, (size[1] + 15) // 16
    tx, ty = rng.integers(0, tiles_x, n), rng.integers(0, tiles_y, n)
    depth = np.exp(rng.uniform(np.log(lo), np.log(hi), n)).astype(np.float32)
    depth[::5] = depth[0]  # ties, broken by the entry's position
    p = np.zeros((n, 15), np.float32)
    p[:, 0], p[:, 1] = 16.0 * tx + 8.0, 16.0 * ty + 8.0
    p[:, 2], p[:, 4] = 1.0, 1.0
    p[:, 5], p[:, 6], p[:, 7] = depth, 3.0, 0.5
    p[:, 11], p[:, 12], p[:, 13], p[:, 14] = tx, ty, tx + 1, ty + 1
    proj = G.proj_from_reference(ctx, torch.from_numpy(p).cuda(), *size)
    b = G.bin(ctx, proj, want_keys=True)
    tile = (ty * tiles_x + tx).astype(np.uint64)
    keys = (tile << np.uint64(32)) | depth.view(np.uint32).astype(np.uint64)
    order = np.argsort(keys, kind="stable")
    assert b.num_entries == n
    assert (b.gauss.cpu().numpy().view(np.uint32) == order).all()
    assert (b.keys.cpu().numpy().view(np.uint64) == keys[order]).all()
    start = np.searchsorted(tile[order], np.arange(tiles_x * tiles_y, dtype=np.uint64), "left")
    end = np.searchsorted(tile[order], np.arange(tiles_x * tiles_y, dtype=np.uint64), "right")
    want = np.where((end > start)[:, None], np.stack([start, end], 1), 0)
    assert (b.tile_range.cpu().numpy().view(np.uint32) == want).all()
    for capacity in (n, n + 1234567):
        gauss, ranges, count, flag, _ = G.bin_device(ctx, proj, capacity)
        assert int(flag.item()) == 0 and int(count.item()) == n
        assert (gauss[:n].cpu().numpy().view(np.uint32) == order).all()
        assert (ranges.cpu().numpy().view(np.uint32) == want).all()
