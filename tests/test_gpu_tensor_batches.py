"""The tensor-core kernel's persistent loop over a second batch of a CTA: key stream from the last key-switching chunk
back to the first rotation row, stage and MMA phases carried over, rotations and accumulators reused. Odd and
even digit counts, one and several chunks; a full second batch and one with an absent gate; and MUX, whose two
jobs a round cuts inside the second. Gates of both batches of the first and the last CTA equal the same gates in
a call of their own (the latency form)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS, ROUND = 148, 4 * 148

# (n, gadget bits, digits, key-switch bits, digits): key switch in 8, 16, 8, 2 and 1 chunks
SHAPES = [(65, 8, 8, 5, 13), (40, 5, 13, 8, 8), (129, 1, 64, 7, 10), (300, 7, 10, 8, 8), (513, 7, 10, 1, 64)]


@pytest.fixture(scope="module")
def ctx(hb):
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != SMS:
        pytest.skip("the rounds below are those of 148 SMs")
    c = hb.Context(0)
    yield c
    c.close()


def evaluator(hb, ctx, shape):
    from hasteboots_b200._lib import HbParams
    raw = HbParams.from_buffer_copy(hb.Parameters.preset(1).raw)
    raw.lwe_dim, raw.br_bits, raw.br_len, raw.ks_bits, raw.ks_len = shape
    sk = hb.KeyGen.generate_secret_key(hb.Parameters(raw, "GOLDILOCKS+%s" % (shape,)), 0)
    return sk, hb.Evaluator(sk, ctx)


@pytest.mark.parametrize("shape", SHAPES)
def test_second_batch_of_a_cta(hb, ctx, shape):
    sk, ev = evaluator(hb, ctx, shape)
    try:
        for count in (2 * ROUND, 2 * ROUND - 1):
            bits = np.random.default_rng(count).integers(0, 2, (2, count)).astype(np.uint8)
            c = [sk.encrypt(b, 10000 * i) for i, b in enumerate(bits)]
            out = ev.xor(c[0], c[1])
            pick = np.r_[0:4, ROUND - 4:ROUND, ROUND:ROUND + 4, count - 4:count]
            assert (out[pick] == ev.xor(c[0][pick], c[1][pick])).all(), count
    finally:
        ev.keys.free()


@pytest.mark.parametrize("shape", SHAPES[:2])
def test_mux_cut_inside_its_second_job(hb, ctx, shape):
    sk, ev = evaluator(hb, ctx, shape)
    try:
        for count in (400, ROUND - 1):
            bits = np.random.default_rng(count).integers(0, 2, (3, count)).astype(np.uint8)
            c = [sk.encrypt(b, 10000 * i) for i, b in enumerate(bits)]
            out = ev.mux(*c)
            cut = ROUND - 4 * -(-count // 4)  # gates of the second job in the round
            pick = np.unique(np.clip(np.r_[0:3, cut - 1:cut + 2, count // 2, count - 2:count], 0, count - 1))
            assert (out[pick] == ev.mux(*(x[pick] for x in c))).all(), count
    finally:
        ev.keys.free()
