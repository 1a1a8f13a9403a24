"""The way out of a wait that runs out, in the tensor-core kernel (bootstrap_tc_kernel): with the key copies withheld
(a flag that nothing sets) and a short limit the call returns HB_ERR_TIMEOUT, and the next call on the same
context gives the words it gave before. One batch per CTA and several, one and several key-switching chunks,
the allocation-free MUX, and external products in their only step (592: the CTA's last batch) and before
another batch (1184)."""

import ctypes
import time

import numpy as np
import pytest

from conftest import hb_params_of
from gpu_util import empty_dev, from_dev, ptr, to_dev

pytestmark = pytest.mark.gpu

HB_ERR_TIMEOUT = -4


class withheld:
    """Keys withheld, and a wait limit of about 0.1 ms of SM clocks."""

    def __init__(self, ctx):
        self.ctx = ctx

    def __enter__(self):
        from hasteboots_b200._lib import lib
        assert lib().hb_ctx_set_wait_limit(self.ctx.handle, 200000) == 0
        assert lib().hb_ctx_test_withhold_keys(self.ctx.handle, 1) == 0
        self.t0 = time.perf_counter()

    def __exit__(self, *exc):
        from hasteboots_b200._lib import lib
        lib().hb_ctx_test_withhold_keys(self.ctx.handle, 0)
        lib().hb_ctx_set_wait_limit(self.ctx.handle, 0)
        assert time.perf_counter() - self.t0 < 30


@pytest.mark.parametrize("set_id,count", [(1, 300), (1, 1300), (2, 300), (101, 592)])
def test_gates_time_out_and_context_recovers(hb, set_id, count):
    from hasteboots_b200._lib import HbError
    ctx = hb.Context(0)
    sk = hb.KeyGen.generate_secret_key(hb_params_of(hb, set_id), 0)
    ev = hb.Evaluator(sk, ctx)
    try:
        bits = np.random.default_rng(31).integers(0, 2, (2, count)).astype(np.uint8)
        c0, c1 = sk.encrypt(bits[0], 5 << 20), sk.encrypt(bits[1], 6 << 20)
        ref = ev.nand(c0, c1)
        with withheld(ctx), pytest.raises(HbError) as err:
            ev.nand(c0, c1)
        assert err.value.code == HB_ERR_TIMEOUT
        out = ev.nand(c0, c1)
        assert (out == ref).all()
        assert (sk.decrypt(out) == 1 - (bits[0] & bits[1])).all()
    finally:
        ev.keys.free()
        ctx.close()


def test_noalloc_mux_times_out_and_recovers(hb):
    from hasteboots_b200._lib import check, lib
    ctx = hb.Context(0)
    sk = hb.KeyGen.generate_secret_key(hb_params_of(hb, 1), 0)
    ev = hb.Evaluator(sk, ctx)
    try:
        count = 300
        bits = np.random.default_rng(78).integers(0, 2, (3, count)).astype(np.uint8)
        cs = [sk.encrypt(b, 9000 * (i + 1)) for i, b in enumerate(bits)]
        d = [to_dev(c) for c in cs]
        out = empty_dev(cs[0].shape, cs[0].dtype)
        args = (ctx.handle, ev.keys.handle, d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), out.data_ptr(), count)
        with withheld(ctx):
            assert lib().hb_gate_mux_device_noalloc(*args) == HB_ERR_TIMEOUT
        check(lib().hb_gate_mux_device_noalloc(*args), "mux_noalloc", ctx.handle)
        got = from_dev(out, cs[0].dtype)
        assert (got == ev.mux(*cs)).all()
        assert (sk.decrypt(got) == np.where(bits[0] == 1, bits[1], bits[2])).all()
    finally:
        ev.keys.free()
        ctx.close()


@pytest.mark.parametrize("count", [592, 1184])
def test_external_products_time_out_and_recover(hb, count):
    import torch
    from hasteboots_b200._lib import HbError, MODULUS, check, lib
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("whole rounds of 148 SMs")
    ctx = hb.Context(0)
    try:
        n, bits, length = 1024, 5, 13
        rng = np.random.default_rng(count)
        rgsw = rng.integers(0, MODULUS[1], 2 * length * 2 * n, dtype=np.uint64)
        d_in = to_dev(rng.integers(0, MODULUS[1], (count, 2 * n), dtype=np.uint64))
        h = ctypes.c_void_p()
        check(lib().hb_rgsw_upload(ctx.handle, 1, 10, bits, length, rgsw.ctypes.data_as(ctypes.c_void_p),
                                   ctypes.byref(h)), "rgsw_upload", ctx.handle)

        def product():
            d_out = empty_dev((count, 2 * n), np.uint64)
            check(lib().hb_external_product_device(ctx.handle, 1, 10, bits, length, h, ptr(d_in), ptr(d_out), count),
                  "ext", ctx.handle)
            ctx.synchronize()
            return from_dev(d_out, np.uint64)

        ref = product()
        assert ref.any(axis=1).all()
        with withheld(ctx), pytest.raises(HbError) as err:
            product()
        assert err.value.code == HB_ERR_TIMEOUT
        assert (product() == ref).all()
        lib().hb_rgsw_free(ctx.handle, h)
    finally:
        ctx.close()
