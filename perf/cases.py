"""Workloads whose speed is tracked: gate bootstrapping over the repository's parameter sets, and the
NTT and external-product entry points.

A case is a dict of plain values; its "kind" says which public entry point it goes through:
  gate   Evaluator.nand/and_/... on device tensors, or on host arrays ("host": copies included)
  lut    Evaluator.bootstrap, a caller's LUT polynomial, host arrays
  mixed  Batch: one graph launch of gate jobs over three parameter sets
  ntt    hb_ntt_roundtrip_device, forward and inverse transforms of a batch of polynomials
  ext    hb_external_product_device, a batch of RLWEs times one RGSW
"""

import ctypes

import numpy as np
import torch

from hasteboots_b200 import tfhe
from hasteboots_b200._lib import MODULUS, check, lib

# (preset id, ternary LWE key) of the parameter sets
SETS = {"babybear": (0, False), "goldilocks": (1, False), "zama": (2, False), "default": (3, False),
        "custom": (4, False), "custom_ternary_key": (4, True)}
GATES = ("nand", "and_", "or_", "nor", "xor", "xnor", "majority", "mux")
# gadget (base bits, digits) of the external products: the presets' own, per field
GADGETS = {1: ((5, 13), (8, 8)), 0: ((8, 4), (5, 7)), 2: ((3, 9), (7, 4))}


def listed():
    return [
        # one gate, as the reference's NAND examples run it, from host arrays and back
        {"name": "babybear_one", "kind": "gate", "set": "babybear", "gate": "nand", "count": 1, "host": True},
        {"name": "goldilocks_one", "kind": "gate", "set": "goldilocks", "gate": "nand", "count": 1, "host": False},
        # a word-sized circuit layer: fewer gates than SMs, three inputs
        {"name": "zama_layer", "kind": "gate", "set": "zama", "gate": "majority", "count": 75, "host": False},
        # a layer that leaves a partial wave
        {"name": "goldilocks_layer", "kind": "gate", "set": "goldilocks", "gate": "xor", "count": 333, "host": False},
        # throughput: the batch of the benchmark, in both word sizes
        {"name": "goldilocks_bulk", "kind": "gate", "set": "goldilocks", "gate": "nand", "count": 16384, "host": False},
        {"name": "babybear_bulk", "kind": "gate", "set": "babybear", "gate": "nand", "count": 16384, "host": False},
        # the sets over DefaultFieldU32: many digits of a small base; two layers (MUX) with a chunked
        # key switch; a ternary LWE key
        {"name": "default_batch", "kind": "gate", "set": "default", "gate": "and_", "count": 2500, "host": True},
        {"name": "custom_mux", "kind": "gate", "set": "custom", "gate": "mux", "count": 900, "host": False},
        {"name": "custom_ternary_key", "kind": "gate", "set": "custom_ternary_key", "gate": "nor", "count": 500, "host": False},
        # a queue of jobs of all three 128-bit sets, planned once and launched as one graph
        {"name": "mixed_jobs", "kind": "mixed", "jobs": 24, "largest": 512, "plan": 4},
        # the NTT table trait and the external product on a batch
        {"name": "ntt_roundtrip", "kind": "ntt", "field": 1, "log_n": 10, "count": 4096},
        {"name": "external_product", "kind": "ext", "field": 1, "log_n": 10, "bits": 5, "len": 13, "count": 4096},
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(("gate", "gate", "gate", "gate", "lut", "mixed", "ntt", "ext"))
    if kind in ("gate", "lut"):
        name = rng.choice(sorted(SETS))
        most = {"goldilocks": 12000, "zama": 8000, "default": 12000}.get(name, 16384)
        if kind == "lut":
            return {"kind": kind, "set": name, "count": _log_uniform(rng, 1, most // 4)}
        gate = rng.choice(GATES)
        return {"kind": kind, "set": name, "gate": gate, "host": rng.random() < 0.4,
                "count": _log_uniform(rng, 1, most // 4 if gate == "mux" else most)}
    if kind == "mixed":
        return {"kind": kind, "jobs": rng.randint(2, 40), "largest": _log_uniform(rng, 8, 1024),
                "plan": rng.randrange(1 << 16)}
    field, log_n = rng.choice((0, 1, 1, 2)), rng.choice((10, 11))
    count = _log_uniform(rng, 1, 8192)
    if kind == "ntt":
        return {"kind": kind, "field": field, "log_n": log_n, "count": count}
    bits, length = rng.choice(GADGETS[field])
    return {"kind": kind, "field": field, "log_n": log_n, "bits": bits, "len": length, "count": count}


def _params(name):
    preset, ternary = SETS[name]
    p = tfhe.Parameters.preset(preset)
    return p.with_ternary_lwe_key() if ternary else p


def _device(a):
    return torch.from_numpy(a.view(np.int64 if a.dtype.itemsize == 8 else np.int32)).cuda()


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _uniform(rng, field, shape):
    """Canonical field words, uniform."""
    words = rng.integers(0, MODULUS[field], shape, dtype=np.uint64)
    return words if field == 1 else words.astype(np.uint32)


def _inputs(sk, rng, count, n):
    return [sk.encrypt(rng.integers(0, 2, count, dtype=np.uint8)) for _ in range(n)]


def _plan(case):
    """Jobs of a mixed batch: (set, gate, count), counts log-uniform."""
    rng = np.random.default_rng(case["plan"])
    names = ("babybear", "goldilocks", "zama")
    return [(names[i % 3], GATES[int(rng.integers(0, 6))],
             max(1, int(case["largest"] ** rng.random()))) for i in range(case["jobs"])]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    state = {"case": case, "ctx": tfhe.Context()}
    ctx = state["ctx"]
    if kind in ("gate", "lut"):
        sk = tfhe.KeyGen.generate_secret_key(_params(case["set"]), seed)
        state["ev"] = tfhe.Evaluator(sk, ctx)
        if kind == "lut":
            p = sk.params
            state["in"] = _inputs(sk, rng, case["count"], 1)
            state["lut"] = _uniform(rng, p.raw.field_id, p.ring_dimension())
        else:
            cts = _inputs(sk, rng, case["count"], 3 if case["gate"] in ("majority", "mux") else 2)
            state["in"] = cts if case["host"] else [_device(c) for c in cts]
    elif kind == "mixed":
        jobs, evs, state["out"] = [], {}, []
        for name, gate, count in _plan(case):
            if name not in evs:
                sk = tfhe.KeyGen.generate_secret_key(_params(name), seed)
                evs[name] = sk, tfhe.Evaluator(sk, ctx)
            sk, ev = evs[name]
            c0, c1 = (_device(c) for c in _inputs(sk, rng, count, 2))
            state["out"].append(torch.zeros_like(c0))
            jobs.append((ev, gate.rstrip("_"), c0, c1, None, state["out"][-1]))
        state["evs"] = evs
        state["batch"] = tfhe.Batch(ctx, jobs)
    else:
        n = 1 << case["log_n"]
        polys = case["count"] * (2 if kind == "ext" else 1)
        state["in"] = _device(_uniform(rng, case["field"], (polys, n)))
        state["out"] = torch.zeros_like(state["in"])
        if kind == "ext":
            rgsw = _uniform(rng, case["field"], 2 * case["len"] * 2 * n)
            state["rgsw"] = ctypes.c_void_p()
            check(lib().hb_rgsw_upload(ctx.handle, case["field"], case["log_n"], case["bits"], case["len"],
                                       rgsw.ctypes.data_as(ctypes.c_void_p), ctypes.byref(state["rgsw"])),
                  "hb_rgsw_upload", ctx.handle)
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "gate":
        return getattr(state["ev"], case["gate"])(*state["in"])
    if kind == "lut":
        return state["ev"].bootstrap(state["in"][0], state["lut"])
    if kind == "mixed":
        state["batch"].launch()
        return state["out"]
    if kind == "ntt":
        check(lib().hb_ntt_roundtrip_device(ctx.handle, case["field"], case["log_n"], _ptr(state["in"]),
                                            _ptr(state["out"]), case["count"]), "ntt", ctx.handle)
    else:
        check(lib().hb_external_product_device(ctx.handle, case["field"], case["log_n"], case["bits"],
                                               case["len"], state["rgsw"], _ptr(state["in"]),
                                               _ptr(state["out"]), case["count"]), "ext", ctx.handle)
    return state["out"]


def exact(case, seed):
    """A round trip gives its input back. The other outputs are whole words fixed by the inputs and keys."""
    if case["kind"] != "ntt":
        return None
    rng = np.random.default_rng(seed)
    words = _uniform(rng, case["field"], (case["count"], 1 << case["log_n"]))
    return words.view(np.int64 if case["field"] == 1 else np.int32)


def _gate_work(name, count, bootstraps=1):
    """Bytes and operations of count gates of a set: keys and ciphertexts once; two operations per
    modular multiplication of the transforms and products of the blind rotation and the key switch."""
    p = _params(name).raw
    word = 8 if p.field_id == 1 else 4
    n, N, logn = p.lwe_dim, p.ring_dim, p.ring_dim.bit_length() - 1
    pairs = 2 if p.lwe_ternary else 1
    keys = (n * pairs * 2 * p.br_len + p.ks_len) * 2 * N * word
    muls = n * ((2 * p.br_len + 2) * N // 2 * logn + pairs * 4 * p.br_len * N)
    muls += (p.ks_len + 2) * N // 2 * logn + 2 * p.ks_len * N
    return keys + 3 * count * (n + 1) * word, 2 * muls * count * bootstraps


def work(case):
    kind = case["kind"]
    if kind in ("gate", "lut"):
        mux = kind == "gate" and case["gate"] == "mux"
        b, f = _gate_work(case["set"], case["count"], 3 if mux else 1)
    elif kind == "mixed":
        counts = {}
        for name, _, count in _plan(case):
            counts[name] = counts.get(name, 0) + count
        parts = [_gate_work(name, count) for name, count in counts.items()]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    else:
        n, word = 1 << case["log_n"], 8 if case["field"] == 1 else 4
        half = n // 2 * case["log_n"]
        if kind == "ntt":
            b, f = 2 * case["count"] * n * word, 2 * case["count"] * (2 * half + n)
        else:
            b = (4 * case["count"] + 4 * case["len"]) * n * word
            f = 2 * case["count"] * ((2 * case["len"] + 2) * half + 4 * case["len"] * n)
    return {"bytes": b, "flops": f}
