"""Adam::step (src/adam.rs:44-61) over the whole range of its operands: the divisions by the
step's bias corrections take rounded reciprocals inside a range of magnitudes and the operator
outside of it, and zero operands are answered without either. Parameters and moments are the
oracle's bit for bit, from subnormal to infinite, at the first steps and at late ones."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from splatrs_b200 import gpu as G
from splatrs_b200._lib import LearningRates

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = G.Context(0)
    yield c
    c.close()


def _spread(rng, shape, lo, hi, zeros):
    a = np.ldexp(rng.uniform(1.0, 2.0, shape), rng.integers(lo, hi, shape)) * rng.choice((-1.0, 1.0), shape)
    a[rng.random(shape) < zeros] = 0.0
    return a.astype(np.float32)


@pytest.mark.parametrize("step", [1, 2, 50, 5000, 1_000_000])
@pytest.mark.parametrize("lo,hi", [(-40, 10), (-149, 127), (-105, -95), (95, 105)])
def test_adam_range_bit_exact(ctx, step, lo, hi):
    n = 2000
    rng = np.random.default_rng(step + 1000 * (lo + 200))
    with np.errstate(all="ignore"):
        p, g = _spread(rng, (n, 59), -20, 5, 0.1), _spread(rng, (n, 59), lo, hi, 0.3)
        m = _spread(rng, (n, 59), lo, hi, 0.3)
        v = np.abs(_spread(rng, (n, 59), lo, hi, 0.3))
    g[0, :4], m[1, :4], v[2, :4] = (np.inf, -np.inf, np.nan, -0.0), (np.inf, -0.0, np.nan, 0.0), (np.inf, np.nan, 0.0, 0.0)
    lr = LearningRates(0.00016, 0.005, 0.001, 0.025, 0.0025, 0.0025 / 20)
    lr6 = np.array([lr.mean, lr.log_scale, lr.quat, lr.opacity, lr.sh_dc, lr.sh_rest], np.float32)
    t = [G.params_to_planes(ctx, torch.from_numpy(a).cuda(), None) for a in (p, g, m, v)]
    G.adam_step(ctx, *t, n, n, step, lr)
    O.adam_step(p, g, m, v, step - 1, lr6)
    for got, want in ((t[0], p), (t[2], m), (t[3], v)):
        got = G.planes_to_params(ctx, got, n, n).cpu().numpy()
        nan = np.isnan(want)
        assert np.array_equal(np.isnan(got), nan)
        assert np.array_equal(got.view(np.uint32)[~nan], want.view(np.uint32)[~nan])


@pytest.mark.parametrize("rate", [1e-30, 1.0, 1e6, 1e25, 3e38])
def test_adam_rate_bit_exact(ctx, rate):
    """Rates and moments whose step overflows to an infinity, or is lost, are the oracle's too."""
    n = 2000
    rng = np.random.default_rng(17)
    p, g = _spread(rng, (n, 59), -20, 5, 0.1), np.zeros((n, 59), np.float32)
    m, v = _spread(rng, (n, 59), -60, 60, 0.1), np.abs(_spread(rng, (n, 59), -60, 60, 0.5))
    lr = LearningRates(*[rate] * 6)
    t = [G.params_to_planes(ctx, torch.from_numpy(a).cuda(), None) for a in (p, g, m, v)]
    G.adam_step(ctx, *t, n, n, 3, lr)
    with np.errstate(all="ignore"):
        O.adam_step(p, g, m, v, 2, np.full(6, rate, np.float32))
    for got, want in ((t[0], p), (t[2], m), (t[3], v)):
        got = G.planes_to_params(ctx, got, n, n).cpu().numpy()
        nan = np.isnan(want)
        assert np.array_equal(np.isnan(got), nan)
        assert np.array_equal(got.view(np.uint32)[~nan], want.view(np.uint32)[~nan])
