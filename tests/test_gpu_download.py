"""The trainer's read-back of its model and moments into host arrays of the caller, at the sizes
where the number of threads that touch the array's pages changes (one thread per MiB, from two
MiB on, eight at most): the records that went in come out bit for bit, the moments are those of
the first step, nothing around the array is written, whether its pages are new or used and
wherever it starts."""
import ctypes as C

import numpy as np
import pytest

from splatrs_b200 import gpu as G
from splatrs_b200 import scenes

pytestmark = pytest.mark.gpu

RECORD = 59 * 4
MIB = 1 << 20
GUARD = 1500  # floats on both sides: more than a page
NAN_BITS = np.uint32(0x7FC01234)


def host_array(n, shift):
    """(whole array, its n records): NaN everywhere, the records `shift` floats off a page."""
    whole = np.empty(2 * GUARD + 59 * n + 1024, np.float32)
    whole.view(np.uint32)[:] = NAN_BITS
    start = GUARD + (-(whole.ctypes.data // 4 + GUARD)) % 1024 + shift
    return whole, whole[start:start + 59 * n].reshape(n, 59)


def around_is_whole(whole, records):
    a = (records.ctypes.data - whole.ctypes.data) // 4
    bits = whole.view(np.uint32)
    return (bits[:a] == NAN_BITS).all() and (bits[a + records.size:] == NAN_BITS).all()


def ptr(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.mark.parametrize("n", [1, 2 * MIB // RECORD, 2 * MIB // RECORD + 1, 8 * MIB // RECORD, 8 * MIB // RECORD + 1,
                               90001])
@pytest.mark.parametrize("shift", [0, 1, 1023])
def test_read_back(n, shift):
    g = scenes.random_gaussians(np.random.default_rng(n), n, -1.0, 1.0, -4.0, 0.3, 1.0)
    cam = scenes.look_at(16, 16, 20.0, 20.0, (0.0, 0.0, -4.0), (0.0, 0.0, 0.0))
    ctx = G.Context(0)
    trainer = G.Trainer(ctx, g, 1.0, [(cam, np.zeros(16 * 16 * 3, np.uint8))])
    model, moments = ctx.lib.splat_trainer_get_model, ctx.lib.splat_trainer_get_moments
    whole, out = host_array(n, shift)
    for _ in range(2):  # the second time over the first time's records
        G.check(model(trainer.h, ptr(out)), ctx.h)
        assert (out.view(np.uint32) == g.view(np.uint32)).all() and around_is_whole(whole, out)
    fresh = np.empty((n, 59), np.float32)
    G.check(model(trainer.h, ptr(fresh)), ctx.h)
    assert (fresh.view(np.uint32) == g.view(np.uint32)).all()
    trainer.step()
    (whole_m, m), (whole_v, v) = host_array(n, shift), host_array(n, shift)
    G.check(moments(trainer.h, ptr(m), ptr(v)), ctx.h)
    assert around_is_whole(whole_m, m) and around_is_whole(whole_v, v)
    # One step from zero: m = (1 - b1) g and v = (1 - b2) g g, three roundings and two.
    grad = m.astype(np.float64) / np.float64(np.float32(1.0) - np.float32(0.9))
    want = np.float64(np.float32(1.0) - np.float32(0.999)) * grad * grad
    live = want > 1e-36
    assert live.any() and (np.abs(v - want)[live] <= 1e-6 * want[live]).all() and (v[~live] <= 2e-36).all()
    ctx.close()
