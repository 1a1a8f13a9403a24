"""The group size that keys under a ternary LWE key are laid out for before any tuning."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HB_ERR_UNSUPPORTED = -5


@pytest.fixture(scope="module")
def ctx(hb):
    c = hb.Context(0)
    yield c
    c.close()


def ternary(hb, preset, **words):
    from hasteboots_b200._lib import HbParams
    raw = HbParams.from_buffer_copy(hb.Parameters.preset(preset).with_ternary_lwe_key().raw)
    for name, value in words.items():
        setattr(raw, name, value)
    return raw


def test_a_dimension_without_kernels_stays_refused(hb, ctx):
    from hasteboots_b200._lib import lib
    raw = ternary(hb, 3, ring_dim=2048, lwe_dim=4, br_bits=14, br_len=2)
    sizes = [ctypes.c_size_t() for _ in range(5)]
    assert lib().hb_params_sizes(ctypes.byref(raw), *(ctypes.byref(s) for s in sizes)) == 0
    bsk, ksk = (np.zeros(sizes[i].value, np.uint32) for i in (2, 3))
    keys = ctypes.c_void_p()
    rc = lib().hb_keys_upload(ctx.handle, ctypes.byref(raw), bsk.ctypes.data_as(ctypes.c_void_p),
                              ksk.ctypes.data_as(ctypes.c_void_p), ctypes.byref(keys))
    assert rc == HB_ERR_UNSUPPORTED and not keys.value


@pytest.mark.parametrize("words,threads", [(dict(), 64), (dict(br_bits=5, br_len=6), 128),
                                           (dict(br_bits=4, br_len=7), 64), (dict(br_bits=14, br_len=2), 128)])
def test_default_group_size_follows_the_digits(hb, ctx, words, threads):
    """DEFAULT_TERNARY with its nine digits, and around the rule's line. Gates under both layouts give the same words."""
    from hasteboots_b200._lib import check, lib
    sk = hb.KeyGen.generate_secret_key(hb.Parameters(ternary(hb, 3, lwe_dim=60, **words), "ternary"), 0)
    ev = hb.Evaluator(sk, ctx)
    try:
        t, g = ctypes.c_int(), ctypes.c_int()
        lib().hb_keys_config(ev.keys.handle, ctypes.byref(t), ctypes.byref(g))
        assert (t.value, g.value) == (threads, 4)
        bits = np.random.default_rng(3).integers(0, 2, (2, 200)).astype(np.uint8)
        c = [sk.encrypt(b, 1000 * i) for i, b in enumerate(bits)]
        out = ev.nand(*c)
        check(lib().hb_keys_set_config(ctx.handle, ev.keys.handle, 192 - threads, 4), "config", ctx.handle)
        assert (ev.nand(*c) == out).all()
    finally:
        ev.keys.free()
