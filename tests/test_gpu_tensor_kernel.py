"""The tensor-core form of the batched Goldilocks kernel (bootstrap_tc_kernel, T = 128 and G = 4) against the
butterfly form (one gate per launch): the outputs of the first and the last CTA equal, and sampled outputs
equal to the oracle's. Gadget and key-switch shapes with odd and even digit counts, one digit, the
smallest and the largest bases it takes and one it leaves to the other form; one and several key-switching
chunks; a full wave of CTAs with an absent gate and one gate more."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (n, gadget bits, digits, key-switch bits, digits)
SHAPES = [(65, 8, 8, 5, 13), (40, 5, 13, 8, 8), (129, 1, 64, 7, 10), (513, 7, 10, 1, 64), (33, 12, 6, 5, 13),
          (70, 3, 22, 16, 4)]


@pytest.fixture(scope="module")
def ctx(hb):
    c = hb.Context(0)
    yield c
    c.close()


def evaluator(hb, ctx, shape):
    from hasteboots_b200._lib import HbParams
    raw = HbParams.from_buffer_copy(hb.Parameters.preset(1).raw)
    raw.lwe_dim, raw.br_bits, raw.br_len, raw.ks_bits, raw.ks_len = shape
    params = hb.Parameters(raw, "GOLDILOCKS+%s" % (shape,))
    sk = hb.KeyGen.generate_secret_key(params, 0)
    return sk, hb.Evaluator(sk, ctx)


@pytest.mark.parametrize("shape", SHAPES)
def test_tensor_form_equals_butterfly_form(hb, ctx, shape):
    from gpu_util import empty_dev, from_dev, to_dev
    from hasteboots_b200._lib import check, lib
    sk, ev = evaluator(hb, ctx, shape)
    try:
        for count in (4 * 148 - 1, 4 * 148 + 1):
            bits = np.random.default_rng(count).integers(0, 2, (2, count)).astype(np.uint8)
            c = [sk.encrypt(b, 10000 * i) for i, b in enumerate(bits)]
            pick = np.r_[0:6, count - 6:count]  # the first and the last CTA
            d = [to_dev(x[pick]) for x in c]
            ref = empty_dev(c[0][pick].shape, c[0].dtype)
            for gate, name in ((0, "nand"), (4, "xor")):
                out = getattr(ev, name)(c[0], c[1])
                check(lib().hb_gate_device_plain(ctx.handle, ev.keys.handle, gate, d[0].data_ptr(), d[1].data_ptr(),
                                                 ref.data_ptr(), len(pick)), "plain", ctx.handle)
                ctx.synchronize()
                assert (out[pick] == from_dev(ref, out.dtype)).all(), name
    finally:
        ev.keys.free()


@pytest.mark.parametrize("pid", [1, 2])
def test_tensor_form_vs_oracle(hb, oracle, oracle_keys, ctx, pid):
    sk = hb.KeyGen.generate_secret_key(hb.Parameters.preset(pid), 0)
    ev = hb.Evaluator(sk, ctx)
    try:
        count = 149  # one gate more than the latency form takes
        bits = np.random.default_rng(7).integers(0, 2, (2, count)).astype(np.uint8)
        c0, c1 = sk.encrypt(bits[0], 500), sk.encrypt(bits[1], 900)
        # extreme coefficients: zero, the largest residue, all equal (rotations by zero and by N)
        c0[0, :-1], c1[0, :-1] = 0, 0
        c0[1, :-1], c1[1, :-1] = oracle.MODULUS[1] - 1, 0
        c0[2, :-1], c1[2, :-1] = oracle.MODULUS[1] // 2, 0
        out = ev.nand(c0, c1)
        pick = [0, 1, 2, 3, 77, 147, 148]
        assert (out[pick] == oracle.gate(oracle_keys(pid), "nand", c0[pick], c1[pick])).all()
        assert (sk.decrypt(out[3:]) == 1 - (bits[0] & bits[1])[3:]).all()
    finally:
        ev.keys.free()
