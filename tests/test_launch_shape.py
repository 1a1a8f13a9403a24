"""The shape of a launch over a list of jobs (hasteboots_b200/csrc/hb_shape.h), whose batches do not span jobs, against
the measured times of a batch. Over GOLDILOCKS no list of jobs may take longer than in the butterfly form alone (the
tensor-core form lasts four gates whether they are there or not, so launches of jobs of one or two gates must not
go to it); over the 32-bit fields none longer than in the best of the compiled variants."""

import os
import random
import subprocess
import tempfile

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hasteboots_b200", "csrc")
SMS = 148

# ms of a CTA's batch by its gates, B200
GOLDILOCKS = {1: 28.7, 2: 38.3, 3: 50.0, 4: 63.7}
TENSOR = 45.8
DEFAULT = {1: 26.0, 2: 26.4, 3: 32.1, 4: 32.2, 5: 43.9, 6: 43.9, 7: 57.0, 8: 57.0}
BABYBEAR = {1: 12.0, 2: 12.1, 3: 15.3, 4: 15.4, 5: 19.6, 6: 19.9, 7: 23.7, 8: 23.7}

DRIVER = r"""
#include <cstdio>
#include "hb_shape.h"
int main() {
  unsigned sms, threads, tuned, nv, tensor, latency, n;
  while (scanf("%u %u %u %u %u %u", &sms, &threads, &tuned, &tensor, &latency, &nv) == 6) {
    std::vector<int> v(nv);
    for (int &x : v) if (scanf("%d", &x) != 1) return 1;
    if (scanf("%u", &n) != 1) return 1;
    std::vector<uint32_t> c(n);
    for (uint32_t &x : c) if (scanf("%u", &x) != 1) return 1;
    const hb::LaunchShape s = hb::launch_shape(c, sms, (int)tuned, v, (int)threads, tensor != 0, latency != 0);
    printf("%d %d\n", s.gates_per_cta, (int)s.tensor);
  }
}
"""


@pytest.fixture(scope="module")
def shape():
    d = tempfile.mkdtemp()
    src, exe = os.path.join(d, "s.cpp"), os.path.join(d, "s")
    open(src, "w").write(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-O1", "-I", CSRC, src, "-o", exe], check=True)

    def run(lists, threads, tuned, variants, tensor=False, latency=True, sms=SMS):
        text = "".join("%d %d %d %d %d %d %s\n%d %s\n" % (sms, threads, tuned, tensor, latency, len(variants),
                                                         " ".join(map(str, variants)), len(c), " ".join(map(str, c)))
                       for c in lists)
        out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split()
        assert len(out) == 2 * len(lists)
        return [(int(g), t == "1") for g, t in zip(out[::2], out[1::2])]
    return run


def job_lists():
    rng = random.Random(5)
    lists = [[1] * 300, [2] * 300, [1] * 149, [3] * 300, [1], [1, 1], [2, 2], [5, 5], [30] * 40, [16384], [593], [5] * 300,
             [8, 8], [100, 100], [296, 296], [600, 600], [1, 4] * 150, [4, 1, 1] * 100]
    for _ in range(400):
        top = rng.choice((1, 2, 3, 4, 8, 40))
        lists.append([rng.randint(1, top) for _ in range(rng.randint(1, 900))])
    return lists


def ms(counts, g, batch):
    """A persistent grid: CTA i takes batches i, i + SMS, ..."""
    costs = [batch[min(g, c - at)] for c in counts for at in range(0, c, g)]
    return max(sum(costs[i::SMS]) for i in range(min(SMS, len(costs))))


@pytest.mark.parametrize("latency", [True, False])
def test_small_jobs_do_not_wait_for_absent_gates(shape, latency):
    lists = job_lists()
    for counts, (g, tensor) in zip(lists, shape(lists, 128, 4, [3, 4], True, latency)):
        if latency and sum(counts) <= SMS:
            assert (g, tensor) == (1, False)
            continue
        now = ms(counts, g, dict.fromkeys(GOLDILOCKS, TENSOR) if tensor else GOLDILOCKS)
        best = min(ms(counts, 3, GOLDILOCKS), ms(counts, 4, GOLDILOCKS), ms(counts, 4, dict.fromkeys(GOLDILOCKS, TENSOR)))
        assert now <= 1.05 * best, (g, tensor, len(counts), sum(counts))  # 5 %: the rule's whole numbers
    # in the tensor-core form they would
    assert ms([1] * 300, 4, dict.fromkeys(GOLDILOCKS, TENSOR)) > 1.5 * ms([1] * 300, 4, GOLDILOCKS)


def test_full_batches_take_the_tensor_form(shape):
    lists = [[592], [300], [30] * 40, [16384], [3] * 200, [400, 400]]
    assert shape(lists, 128, 4, [3, 4], True) == [(4, True)] * len(lists)
    assert not any(tensor for _, tensor in shape(lists, 128, 4, [3, 4], False))


@pytest.mark.parametrize("batch,variants", [(DEFAULT, [4, 6, 8]), (DEFAULT, [4, 8]), (BABYBEAR, [4, 6, 8]), (BABYBEAR, [6])])
def test_variant_of_the_32_bit_fields(shape, batch, variants):
    lists = job_lists()
    for counts, (g, tensor) in zip(lists, shape(lists, 64, variants[-1], variants, False, False)):
        assert not tensor
        assert ms(counts, g, batch) <= 1.10 * min(ms(counts, v, batch) for v in variants), (g, counts[:9], len(counts))


def test_edges(shape):
    # the one-gate form where every gate has an SM; keys tuned to it keep it
    assert shape([[148], [1] * 148, [149]], 64, 8, [4, 6, 8]) == [(1, False), (1, False), (4, False)]
    assert shape([[5000]], 64, 1, [4, 6, 8]) == [(1, False)]
    # variants beyond the tuned one are not taken, in any order
    assert shape([[5000]], 64, 6, [8, 6, 4]) == [(6, False)]
    assert shape([[5000], [2]], 64, 6, [6, 4], sms=1) == [(6, False), (4, False)]
