"""photometric_loss (src/loss.rs:137-190) at the edges of its two kernels' tiles and of the line
between them: the gradient bit-identical to the oracle's, loss, SSIM and PSNR to summation
order, from 8-bit targets of every value."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from splatrs_b200 import gpu as G

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = G.Context(0)
    yield c
    c.close()


# 1024 x 576 has 576 tiles of 32 x 32 (the small kernels on 148 SMs), 1024 x 608 has 608.
@pytest.mark.parametrize("w,h", [(1, 1), (5, 3), (31, 15), (32, 16), (33, 17), (37, 65), (1024, 576), (1024, 608)])
@pytest.mark.parametrize("u8", [True, False])
def test_loss_at_the_edges_of_its_tiles(ctx, w, h, u8):
    rng = np.random.default_rng(w * 10000 + h)
    pred = rng.uniform(-0.2, 1.2, w * h * 3).astype(np.float32)
    t8 = (np.arange(w * h * 3) * 37 % 256).astype(np.uint8)
    target = t8.astype(np.float32) / np.float32(255.0) if u8 else rng.uniform(0, 1, w * h * 3).astype(np.float32)
    out, grad = G.photometric_loss(ctx, torch.from_numpy(pred).cuda(),
                                   torch.from_numpy(t8 if u8 else target).cuda(), w, h, 0.2)
    loss, want = O.photometric_loss(pred, target, w, h, 0.2)
    assert np.array_equal(grad.cpu().numpy(), want)
    o = out.cpu().numpy()
    assert abs(o[0] - loss) <= 2e-6 * max(1.0, abs(loss))
    assert abs(o[2] - O.psnr(pred, target)) < 1e-3
