"""The caller's scratch of the device-driven sort (splat_bin_sort_device): any alignment, scratch
for one capacity serves every smaller one, and nothing is written outside of the bytes that
splat_bin_sort_device_scratch_bytes asks for."""
import numpy as np
import pytest
import torch

from splatrs_b200 import _lib
from splatrs_b200 import gpu as G

GUARD = 4 << 20


def need(capacity):
    return int(_lib.lib().splat_bin_sort_device_scratch_bytes(capacity))


def sort_in(ctx, n, capacity, offset, size):
    """Sorts n one-tile Gaussians in scratch bytes [offset, offset + size) of a patterned buffer;
    the sorted Gaussians, those of the host-driven sort and whether the pattern around is whole."""
    rng = np.random.default_rng(n)
    w, h = 640, 480
    tx, ty = rng.integers(0, w // 16, n), rng.integers(0, h // 16, n)
    p = np.zeros((n, 15), np.float32)
    p[:, 0], p[:, 1] = 16.0 * tx + 8.0, 16.0 * ty + 8.0
    p[:, 2], p[:, 4], p[:, 5] = 1.0, 1.0, rng.uniform(0.5, 9.0, n)
    p[:, 6], p[:, 7] = 3.0, 0.5
    p[:, 11], p[:, 12], p[:, 13], p[:, 14] = tx, ty, tx + 1, ty + 1
    proj = G.proj_from_reference(ctx, torch.from_numpy(p).cuda(), w, h)
    want = G.bin(ctx, proj)
    buf = torch.full((offset + size + GUARD,), 0xA5, dtype=torch.uint8, device="cuda")
    assert buf.data_ptr() % 256 == 0
    scratch = buf[offset:offset + size]
    gauss, ranges, count, flag, used = G.bin_device(ctx, proj, capacity, scratch)
    assert used is scratch and int(flag.item()) == 0 and int(count.item()) == n
    assert torch.equal(ranges, want.tile_range)
    whole = bool((buf[:offset] == 0xA5).all()) and bool((buf[offset + size:] == 0xA5).all())
    return gauss[:n], want.gauss, whole


@pytest.mark.gpu
@pytest.mark.parametrize("n,capacity", [(1, 1), (999, 1003), (65536, 65536), (70001, 70003), (786433, 786433)])
@pytest.mark.parametrize("offset", [8, 16, 4, 129, 248])
def test_scratch_at_any_alignment(n, capacity, offset):
    ctx = G.Context(0)
    got, want, whole = sort_in(ctx, n, capacity, offset, need(capacity))
    assert torch.equal(got, want) and whole
    ctx.close()


def test_scratch_never_shrinks_with_the_capacity():
    edges = [c + d for c in (0, 1, 1024, 2048, 4096, 1 << 16, 1 << 17, 3 << 18, 3 << 19, 1 << 30) for d in (-1, 0, 1)]
    sizes = sorted({c for c in edges if c >= 0} | set(range(1, 2_000_000, 997)) | {800_000, 830_000})
    asked = [need(c) for c in sizes]
    assert all(a <= b for a, b in zip(asked, asked[1:]))


@pytest.mark.gpu
@pytest.mark.parametrize("capacity,larger", [(65536, 65537), (65536, 70000), (786432, 786433), (786432, 800000)])
def test_scratch_of_a_larger_capacity(capacity, larger):
    ctx = G.Context(0)
    got, want, whole = sort_in(ctx, capacity, capacity, 0, need(larger))
    assert torch.equal(got, want) and whole
    ctx.close()
