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
