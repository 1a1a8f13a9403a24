"""External products over Goldilocks with one to four digits, at the batch sizes where the form changes (whole rounds of
four RLWEs per SM with no, one, two, three and more after them): sampled products equal the oracle's."""

import ctypes

import numpy as np
import pytest

from gpu_util import empty_dev, from_dev, ptr, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [1, 2, 3, 4])
def test_few_digits(hb, oracle, length):
    from hasteboots_b200._lib import check, lib
    ctx = hb.Context(0)
    try:
        n, bits, q = 1024, 8, oracle.MODULUS[1]
        rng = np.random.default_rng(length)
        rgsw = rng.integers(0, q, 2 * length * 2 * n, dtype=np.uint64)
        rl = rng.integers(0, q, (2963, 2 * n), dtype=np.uint64)
        rl[0], rl[1] = 0, q - 1
        h = ctypes.c_void_p()
        check(lib().hb_rgsw_upload(ctx.handle, 1, 10, bits, length, rgsw.ctypes.data_as(ctypes.c_void_p),
                                   ctypes.byref(h)), "rgsw_upload", ctx.handle)
        d_in = to_dev(rl)
        for count in (1, 297, 592, 593, 594, 595, 889, 1186, 2961, 2963):
            d_out = empty_dev(rl.shape, np.uint64)
            check(lib().hb_external_product_device(ctx.handle, 1, 10, bits, length, h, ptr(d_in), ptr(d_out), count),
                  "ext", ctx.handle)
            ctx.synchronize()
            out = from_dev(d_out, np.uint64)
            pick = sorted({i for i in (0, 1, 147, 591, 592, 593, 1184, count - 1) if i < count})
            assert (out[pick] == oracle.external_product(1, 10, bits, length, rl[pick], rgsw)).all(), count
            assert not out[count:].any()
        lib().hb_rgsw_free(ctx.handle, h)
    finally:
        ctx.close()
