"""A launch that CUDA refuses is reported by the call that made it and by no later one."""
import pytest
import torch

from splatrs_b200 import gpu as G
from splatrs_b200._lib import LearningRates, SplatError

pytestmark = pytest.mark.gpu


def test_refused_launch_is_reported_once():
    ctx = G.Context(0)
    height = 32 * 65535 + 1  # one row of blocks more than a grid holds: refused on the host
    image = torch.zeros(3 * height, device="cuda")
    with pytest.raises(SplatError):
        G.photometric_loss(ctx, image, image, 1, height, 0.2)
    p, g, m, v = (G.empty_planes(64) for _ in range(4))
    G.adam_step(ctx, p, g, m, v, 64, 64, 1, LearningRates(0.1, 0.1, 0.1, 0.1, 0.1, 0.1))
    torch.cuda.synchronize()
    ctx.close()
