"""The trainer's read-back of its model at the edges of the download's chunks: the records that
went in come out bit for bit, into new and into used host arrays, and the moments are zero."""
import numpy as np
import pytest

from splatrs_b200 import gpu as G
from splatrs_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 8191, 8192, 8193, 4 * 8192, 4 * 8192 + 1, 11 * 8192 + 77])
def test_model_round_trip(n):
    g = scenes.random_gaussians(np.random.default_rng(n), n, -1.0, 1.0, -4.0, 0.3, 1.0)
    cam = scenes.look_at(16, 16, 20.0, 20.0, (0.0, 0.0, -4.0), (0.0, 0.0, 0.0))
    ctx = G.Context(0)
    trainer = G.Trainer(ctx, g, 1.0, [(cam, np.zeros(16 * 16 * 3, np.uint8))])
    for _ in range(2):
        assert (trainer.model().view(np.uint32) == g.view(np.uint32)).all()
    m, v = trainer.moments()
    assert not m.any() and not v.any()
    ctx.close()
