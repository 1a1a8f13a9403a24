"""The latency form over 64-bit keys laid out for 64 threads a gate (whose key words are prefetched) and for 128: one
gate in a cluster and one gate per SM give the same words."""

import numpy as np
import pytest

from conftest import hb_params_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("set_id", [1, 2])
def test_both_layouts_give_the_same_words(hb, set_id):
    from hasteboots_b200._lib import check, lib
    ctx = hb.Context(0)
    sk = hb.KeyGen.generate_secret_key(hb_params_of(hb, set_id), 0)
    ev = hb.Evaluator(sk, ctx)
    try:
        bits = np.random.default_rng(set_id).integers(0, 2, (2, 100)).astype(np.uint8)
        c = [sk.encrypt(b, 500 * (i + 1)) for i, b in enumerate(bits)]
        out = {}
        for t in (128, 64):
            check(lib().hb_keys_set_config(ctx.handle, ev.keys.handle, t, 4), "config", ctx.handle)
            out[t] = ev.nand(c[0][:1], c[1][:1]), ev.nand(*c)
        assert (out[64][0] == out[128][0]).all() and (out[64][1] == out[128][1]).all()
        assert (sk.decrypt(out[64][1]) == 1 - (bits[0] & bits[1])).all()
    finally:
        ev.keys.free()
        ctx.close()
