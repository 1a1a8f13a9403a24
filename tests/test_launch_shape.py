"""The shape of a launch over a list of jobs (hasteboots_b200/csrc/hb_shape.h), whose batches do not span jobs, against
the measured times of a batch. Over GOLDILOCKS no list of jobs may take longer than in the butterfly form alone (the
tensor-core form lasts four gates whether they are there or not, so launches of jobs of one or two gates must not
go to it); over the 32-bit fields none longer than in the best of the compiled variants. And external products over
GOLDILOCKS, by digits and number of RLWEs."""

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
#include <cstdlib>
#include "hb_shape.h"
int main(int argc, char **argv) {
  if (argc == 4) {
    printf("%zu\n", hb::external_products_by_butterflies(strtoull(argv[1], 0, 10), (uint32_t)atoi(argv[2]), strtoull(argv[3], 0, 10)));
    return 0;
  }
  unsigned sms, threads, tuned, nv, tensor, latency, shared, n;
  while (scanf("%u %u %u %u %u %u %u", &sms, &threads, &tuned, &tensor, &latency, &shared, &nv) == 7) {
    std::vector<int> v(nv);
    for (int &x : v) if (scanf("%d", &x) != 1) return 1;
    if (scanf("%u", &n) != 1) return 1;
    std::vector<uint32_t> c(n);
    for (uint32_t &x : c) if (scanf("%u", &x) != 1) return 1;
    const hb::LaunchShape s = hb::launch_shape(c, sms, (int)tuned, v, (int)threads, tensor != 0, latency != 0, shared != 0);
    printf("%d %d\n", s.gates_per_cta, (int)s.tensor);
  }
}
"""


@pytest.fixture(scope="module")
def exe():
    d = tempfile.mkdtemp()
    src, exe = os.path.join(d, "s.cpp"), os.path.join(d, "s")
    open(src, "w").write(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-O1", "-I", CSRC, src, "-o", exe], check=True)
    return exe


@pytest.fixture(scope="module")
def shape(exe):

    def run(lists, threads, tuned, variants, tensor=False, latency=True, sms=SMS, shared=False):
        text = "".join("%d %d %d %d %d %d %d %s\n%d %s\n" % (sms, threads, tuned, tensor, latency, shared, len(variants),
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


def total(counts, g, batch):
    return sum(batch[min(g, c - at)] for c in counts for at in range(0, c, g))


def test_among_other_launches(shape):
    """The form that holds SMs for less, and gates per CTA from the number of gates alone."""
    lists = job_lists()
    tensor_batch = dict.fromkeys(GOLDILOCKS, TENSOR)
    for counts, (g, tensor) in zip(lists, shape(lists, 128, 4, [3, 4], True, shared=True)):
        if sum(counts) > SMS:
            best = min(total(counts, 4, GOLDILOCKS), total(counts, 4, tensor_batch))
            assert total(counts, g, tensor_batch if tensor else GOLDILOCKS) <= 1.10 * best
    baby = [24, 10, 278, 463, 44, 2, 8, 350]
    assert shape([baby], 64, 8, [4, 6, 8], shared=True) == [(8, False)]
    assert total(baby, 8, BABYBEAR) < total(baby, 6, BABYBEAR)
    lists = [[148], [200], [592], [600], [888], [1184], [1185], [1] * 300]
    assert [g for g, _ in shape(lists, 64, 8, [4, 6, 8], shared=True)] == [1, 4, 4, 6, 6, 8, 8, 4]


def test_edges(shape):
    # the one-gate form where every gate has an SM; keys tuned to it keep it
    assert shape([[148], [1] * 148, [149]], 64, 8, [4, 6, 8]) == [(1, False), (1, False), (4, False)]
    assert shape([[5000]], 64, 1, [4, 6, 8]) == [(1, False)]
    # variants beyond the tuned one are not taken, in any order
    assert shape([[5000]], 64, 6, [8, 6, 4]) == [(6, False)]
    assert shape([[5000], [2]], 64, 6, [6, 4], sms=1) == [(6, False), (4, False)]


# us of one call on B200 by digits and RLWEs: all in the butterfly form, and the whole rounds in the tensor-core form
# with a rest of at most two per SM in a launch of its own
EXTERNAL = {
    1: {592: (25.1, 29.6), 593: (33.3, 46.8), 740: (45.6, 46.7), 1184: (45.5, 53.7), 1185: (53.6, 70.0), 4096: (164, 199)},
    2: {592: (35.3, 33.2), 593: (47.7, 53.6), 594: (51.5, 53.5), 596: (63.7, 53.5), 740: (64.0, 53.7), 888: (64.1, 57.7),
        1184: (64.2, 59.8), 1185: (77.4, 80.1), 1188: (92.5, 80.1), 2369: (137, 149), 2372: (152.5, 148.1),
        2961: (170, 191), 2964: (184.5, 190.9), 3553: (204, 226), 4096: (237, 218), 4148: (247, 256), 8192: (469, 426)},
    3: {592: (45.5, 41.4), 593: (61.7, 65.8), 594: (66.0, 65.8), 596: (82.3, 65.8), 888: (87.7, 70.1), 1188: (121.5, 100.9),
        2369: (181, 187), 2372: (202, 187), 2961: (226, 239), 2964: (244, 238), 3556: (285, 281), 4096: (315, 279)},
    4: {592: (53.9, 43.6), 593: (74.2, 74.1), 740: (107, 73.7), 1185: (123, 111), 2369: (224, 202), 4096: (389, 298)},
    13: {592: (153, 100), 593: (214, 180), 700: (302, 179), 1184: (312, 213), 4096: (1012, 693)},
}


@pytest.mark.parametrize("digits", sorted(EXTERNAL))
def test_form_of_external_products(exe, digits):
    def rest(count):
        return int(subprocess.run([exe, str(count), str(digits), str(SMS)], capture_output=True, text=True, check=True).stdout)
    for count, (butterfly, tensor) in EXTERNAL[digits].items():
        assert (butterfly if rest(count) == count else tensor) <= 1.01 * min(butterfly, tensor), count
    for count in (1, 2, 148, 296, 297, 592, 593, 888, 889, 1184, 100000):
        r, whole = rest(count), 4 * SMS
        assert r == count or r <= 2 * SMS and ((count - r) % whole == 0 or r == 0)
        if digits >= 4:
            assert r == (count % whole if count % whole <= 2 * SMS else 0)
