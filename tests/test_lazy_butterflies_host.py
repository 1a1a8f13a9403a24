"""The unreduced butterflies of the transforms over DefaultFieldU32 (Mont32::ct_lazy, gs_lazy, tame), compiled
for the host: residues and bounds at the extreme words, forward over 11 stages from canonical words and
inverse over a pass of four stages from words below 2P."""

import os
import random
import subprocess
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
P = 132120577

DRIVER = r"""
#include <cstdio>
#include "hb_field.cuh"
using F = hb::DefaultFieldU32;
int main() {
  static_assert(F::LAZY && !hb::BabyBear::LAZY, "lazy fields");
  unsigned x, y, w, bound;
  // "x y w bound": CT and GS butterflies of (x, y) with twiddle w, and tame(x)
  while (scanf("%u %u %u %u", &x, &y, &w, &bound) == 4) {
    const F::Tw t = F::make_tw(w);
    unsigned cx = x, cy = y, gx = x, gy = y;
    F::ct_lazy(cx, cy, t);
    F::gs_lazy(gx, gy, t, bound);
    printf("%u %u %u %u %u\n", cx, cy, gx, gy, F::tame(x));
  }
  return 0;
}
"""


def test_lazy_butterflies_keep_residues_and_bounds():
    d = tempfile.mkdtemp()
    src, exe = os.path.join(d, "lazy.cpp"), os.path.join(d, "lazy")
    open(src, "w").write(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "hasteboots_b200", "csrc"), src, "-o", exe],
                   check=True)
    rng = random.Random(3)
    cases = []
    for stage in range(11):  # forward: inputs below (2 stage + 1) P
        top = (2 * stage + 1) * P - 1
        for x in (0, P - 1, top, rng.randrange(top + 1)):
            for y in (0, top, rng.randrange(top + 1)):
                for w in (0, 1, P - 1, rng.randrange(P)):
                    cases.append(("ct", x, y, w, 2 * stage + 1))
    for bound in (2, 4, 8, 16):  # inverse: inputs below bound P
        top = bound * P - 1
        for x in (0, P - 1, top, rng.randrange(top + 1)):
            for y in (0, top, rng.randrange(top + 1)):
                for w in (0, 1, P - 1, rng.randrange(P)):
                    cases.append(("gs", x, y, w, bound))
    for x in (0, P - 1, P, 2 * P - 1, 24 * P - 1, 32 * P - 1, (1 << 32) - 1):
        cases.append(("tame", x, 0, 1, 16))
    text = "".join(f"{x} {y} {w} {b}\n" for _, x, y, w, b in cases)
    out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split("\n")
    for (kind, x, y, w, b), line in zip(cases, out):
        cx, cy, gx, gy, tx = map(int, line.split())
        assert tx % P == x % P and tx < 2 * P
        if kind == "ct":
            assert (cx % P, cy % P) == ((x + w * y) % P, (x - w * y) % P)
            assert max(cx, cy) < (b + 2) * P < 1 << 32
        if kind == "gs":
            assert (gx % P, gy % P) == ((x + y) % P, (x - y) * w % P)
            assert gx < 2 * b * P < 1 << 32 and gy < 2 * P
