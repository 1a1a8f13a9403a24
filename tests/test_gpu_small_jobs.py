"""Batches of many small jobs and small allocation-free MUXes: their gates equal the same gates in a call of their
own, whatever the launch's shape, and over GOLDILOCKS jobs of one gate do not last as long as jobs of four (they
stay in the butterfly form: 87 ms against 137 for 300 jobs; in the tensor-core form both take 137)."""

import time

import numpy as np
import pytest

from conftest import hb_params_of
from gpu_util import empty_dev, from_dev, to_dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(hb):
    c = hb.Context(0)
    yield c
    c.close()


def key(hb, ctx, set_id):
    sk = hb.KeyGen.generate_secret_key(hb_params_of(hb, set_id), 0)
    return sk, hb.Evaluator(sk, ctx)


def jobs_of(ev, sizes, d0, d1, out):
    jobs, at = [], 0
    for n in sizes:
        jobs.append((ev, "nand", d0[at:at + n], d1[at:at + n], None, out[at:at + n]))
        at += n
    return jobs


# one round and several; every mix of the forms' line; GOLDILOCKS, ZAMA, the chunked key switch, 32-bit fields
@pytest.mark.parametrize("set_id,sizes", [(1, [1] * 149), (1, [2] * 80), (1, [1, 4] * 90), (1, [3, 1] * 60), (101, [1] * 160),
                                          (101, [2, 2, 3] * 60), (3, [30] * 40), (0, [5] * 150), (4, [1, 9] * 80)])
def test_batches_of_small_jobs(hb, ctx, set_id, sizes):
    sk, ev = key(hb, ctx, set_id)
    batch = None
    try:
        total = sum(sizes)
        bits = np.random.default_rng(total).integers(0, 2, (2, total)).astype(np.uint8)
        c = [sk.encrypt(b, 40000 * (i + 1)) for i, b in enumerate(bits)]
        d0, d1 = (to_dev(x) for x in c)
        out = empty_dev(c[0].shape, c[0].dtype)
        batch = hb.Batch(ctx, jobs_of(ev, sizes, d0, d1, out))
        batch.launch()
        ctx.synchronize()
        got = from_dev(out, c[0].dtype)
        assert (sk.decrypt(got) == 1 - (bits[0] & bits[1])).all()
        pick = np.r_[0:6, total // 2:total // 2 + 4, total - 6:total]
        assert (got[pick] == ev.nand(c[0][pick], c[1][pick])).all()
    finally:
        if batch:
            batch.free()
        ev.keys.free()


@pytest.mark.parametrize("set_id,count", [(1, 1), (1, 2), (1, 3), (101, 2), (3, 8), (3, 300), (0, 5)])
def test_small_noalloc_mux(hb, ctx, set_id, count):
    from hasteboots_b200._lib import check, lib
    sk, ev = key(hb, ctx, set_id)
    try:
        bits = np.random.default_rng(count).integers(0, 2, (3, count)).astype(np.uint8)
        c = [sk.encrypt(b, 9000 * (i + 1)) for i, b in enumerate(bits)]
        d = [to_dev(x) for x in c]
        out = empty_dev(c[0].shape, c[0].dtype)
        check(lib().hb_gate_mux_device_noalloc(ctx.handle, ev.keys.handle, d[0].data_ptr(), d[1].data_ptr(),
                                               d[2].data_ptr(), out.data_ptr(), count), "mux_noalloc", ctx.handle)
        assert (from_dev(out, c[0].dtype) == ev.mux(*c)).all()
    finally:
        ev.keys.free()


def test_jobs_of_one_gate_do_not_last_four(hb, ctx):
    sk, ev = key(hb, ctx, 1)
    ms, batches = {}, []
    try:
        c = sk.encrypt(np.zeros(1200, np.uint8))
        d = to_dev(c)
        out = empty_dev(c.shape, c.dtype)
        for n in (1, 4):
            batches.append(hb.Batch(ctx, jobs_of(ev, [n] * 300, d, d, out)))
            for _ in range(3):
                t = time.perf_counter()
                batches[-1].launch()
                ctx.synchronize()
                ms[n] = min(ms.get(n, 1e9), time.perf_counter() - t)
        assert ms[1] < 0.8 * ms[4]
    finally:
        for b in batches:
            b.free()
        ev.keys.free()
