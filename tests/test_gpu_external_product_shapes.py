"""External products at the batch sizes where the launch changes: one, two, three and four RLWEs per SM, whole
rounds with and without a rest, over Goldilocks with N = 1024 (tensor-core form for whole rounds), and one
more field and dimension. Sampled products equal the oracle's; edge RLWEs (zero, all Q - 1) are among them."""

import ctypes

import numpy as np
import pytest

from gpu_util import empty_dev, from_dev, ptr, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("field,log_n,bits,length", [(1, 10, 8, 8), (1, 10, 5, 13), (1, 10, 1, 3), (1, 10, 9, 8),
                                                     (1, 11, 8, 8), (0, 10, 8, 4), (2, 11, 7, 4)])
def test_batch_sizes(hb, oracle, field, log_n, bits, length):
    from hasteboots_b200._lib import check, lib
    ctx = hb.Context(0)
    try:
        n, q = 1 << log_n, oracle.MODULUS[field]
        rng = np.random.default_rng(bits)
        dt = oracle.dtype_of(field)
        rgsw = rng.integers(0, q, 2 * length * 2 * n, dtype=np.uint64).astype(dt)
        most = 1185
        rl = rng.integers(0, q, (most, 2 * n), dtype=np.uint64).astype(dt)
        rl[0], rl[1], rl[2, :n], rl[3, n:] = 0, q - 1, 0, q - 1
        h = ctypes.c_void_p()
        check(lib().hb_rgsw_upload(ctx.handle, field, log_n, bits, length, rgsw.ctypes.data_as(ctypes.c_void_p),
                                   ctypes.byref(h)), "rgsw_upload", ctx.handle)
        d_in = to_dev(rl)
        for count in (1, 2, 148, 149, 296, 297, 591, 592, 593, 740, 889, 1185):
            d_out = empty_dev(rl.shape, dt)
            check(lib().hb_external_product_device(ctx.handle, field, log_n, bits, length, h, ptr(d_in), ptr(d_out),
                                                   count), "ext", ctx.handle)
            ctx.synchronize()
            out = from_dev(d_out, dt)
            pick = sorted({i for i in (0, 1, 2, 3, 147, 592, count - 1) if i < count})
            assert (out[pick] == oracle.external_product(field, log_n, bits, length, rl[pick], rgsw)).all(), count
            assert not out[count:].any()
        lib().hb_rgsw_free(ctx.handle, h)
    finally:
        ctx.close()
