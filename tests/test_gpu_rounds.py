"""Gate calls larger than one round of CTAs: the gates after the whole rounds take a second launch of its own
shape. Outputs around every bound equal the outputs of the same gates in calls of their own (the latency
form), for rests of one gate, of one gate per SM and one more, of several gates per SM, of one gate less than
a round, and for the two jobs of MUX, whose rest is cut out of the second."""

import numpy as np
import pytest

from conftest import hb_params_of

pytestmark = pytest.mark.gpu

SMS = 148


@pytest.fixture(scope="module")
def ctx(hb):
    c = hb.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("set_id,tuned", [(0, 8), (4, 8), (100, 4)])
def test_rest_of_the_rounds(hb, ctx, set_id, tuned):
    import ctypes

    import torch
    from hasteboots_b200._lib import lib
    if torch.cuda.get_device_properties(0).multi_processor_count != SMS:
        pytest.skip("the bounds below are those of 148 SMs")
    sk = hb.KeyGen.generate_secret_key(hb_params_of(hb, set_id), 0)
    ev = hb.Evaluator(sk, ctx)
    try:
        t, g = ctypes.c_int(), ctypes.c_int()
        lib().hb_keys_config(ev.keys.handle, ctypes.byref(t), ctypes.byref(g))
        assert g.value == tuned
        rnd = SMS * tuned
        most = 2 * rnd
        bits = np.random.default_rng(set_id).integers(0, 2, (3, most)).astype(np.uint8)
        c = [sk.encrypt(b, 100000 * i) for i, b in enumerate(bits)]
        for count in (rnd + 1, rnd + SMS, rnd + SMS + 1, rnd + 3 * SMS, 2 * rnd - 1, SMS + 1, 3 * SMS, rnd - 1):
            out = ev.xor(c[0][:count], c[1][:count])
            pick = np.unique(np.clip(np.r_[0, 1, SMS - 1, SMS, rnd - 1, rnd, rnd + 1, count - 2, count - 1], 0, count - 1))
            assert (out[pick] == ev.xor(c[0][pick], c[1][pick])).all(), count
        count = rnd - 100  # 2 count gates in the first layer: one round and a rest
        out = ev.mux(*(x[:count] for x in c))
        pick = np.unique(np.clip(np.r_[0, SMS, rnd - count - 1, rnd - count, count // 2, count - 1], 0, count - 1))
        assert (out[pick] == ev.mux(*(x[pick] for x in c))).all()
        assert (sk.decrypt(out) == np.where(bits[0, :count], bits[1, :count], bits[2, :count])).all()
    finally:
        ev.keys.free()


@pytest.mark.parametrize("set_id", [0, 1])
def test_device_calls_take_nothing_from_the_budget(hb, set_id):
    """Once the keys are there a gate call, of one launch or of two, fits whatever the budget leaves."""
    from gpu_util import empty_dev, from_dev, to_dev
    from hasteboots_b200._lib import check, lib
    sk = hb.KeyGen.generate_secret_key(hb_params_of(hb, set_id), 0)
    ctx = hb.Context(0, hbm_budget=1 << 30)
    ev = hb.Evaluator(sk, ctx)
    try:
        used = ctx.hbm_in_use()
        bits = np.random.default_rng(5).integers(0, 2, (2, 1300)).astype(np.uint8)
        c = [sk.encrypt(b, 5000 * i) for i, b in enumerate(bits)]
        d = [to_dev(x) for x in c]
        out = empty_dev(c[0].shape, c[0].dtype)
        for count in (1, 149, 700, 1300):
            check(lib().hb_gate_device(ctx.handle, ev.keys.handle, 0, d[0].data_ptr(), d[1].data_ptr(), None,
                                       out.data_ptr(), count), "gate", ctx.handle)
            ctx.synchronize()
            assert ctx.hbm_in_use() == used, count
        assert (sk.decrypt(from_dev(out, c[0].dtype)) == 1 - (bits[0] & bits[1])).all()
    finally:
        ev.keys.free()
        ctx.close()
