"""The handovers of the tensor-core bootstrapping kernel (hasteboots_b200/csrc/hb_handover.h): compute warps arrive
at a named barrier and go on, the MMA and the key warp wait at it. A model of that protocol, with the barrier of
every handover taken from the header, is run through every interleaving: no warp may arrive twice at a barrier
before it completed once, every warp must come to its end, and the auxiliary warps must meet the same handovers
as the compute warps, also where the compute warps stop after a step. With a single barrier the model finds the
double arrival."""

import os
import subprocess
import tempfile

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hasteboots_b200", "csrc")

COMPUTE, MMA, KEY = 2, 2, 3  # agents 0 and 1 stand for the compute warps, then the MMA warp and the key warp


@pytest.fixture(scope="module")
def barriers():
    d = tempfile.mkdtemp()
    src, exe = os.path.join(d, "h.cpp"), os.path.join(d, "h")
    open(src, "w").write('#include <cstdio>\n#include "hb_handover.h"\n'
                         "int main() { for (unsigned k = 0; k < 130; ++k) printf(\"%d\\n\", hb::tc_handover_barrier(k)); }\n")
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, src, "-o", exe], check=True)
    return [int(x) for x in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()]


def programs(barrier, steps, units, stop_after):
    """Operations of every agent. A step: handover 0, then handovers 1 .. units + 1, and before handover u + 1 the
    compute warps wait for the MMA group issued after handover u (all but the last have one); at its end they
    meet each other. stop_after: the compute warps stop after that step, and tell so at one more handover."""
    compute, mma, key = [], [], []
    groups = 0
    for step in range(steps):
        for k in range(units + 2):
            if step <= (stop_after if stop_after is not None else steps):
                if k > 0:
                    compute.append(("group", groups + k))
                compute.append(("arrive", barrier(k)))
            mma.append(("sync", barrier(k), step))
            if k <= units:
                mma.append(("issue",))
            key.append(("sync", barrier(k), step))
        groups += units + 1
        compute.append(("meet",))
        if stop_after == step:
            if step + 1 < steps:
                compute.append(("arrive", barrier(0)))
            break
    if stop_after is not None and stop_after + 1 < steps:  # the auxiliary warps leave at the next step's handover 0
        for p in (mma, key):
            p.append(("sync", barrier(0), stop_after + 1))
    return [compute, compute, mma, key]


def explore(progs):
    """Every interleaving: "double arrival", "stuck" or "ok". A state: each agent's place, MMA groups issued, and per
    barrier the agents that arrived since it last completed."""
    ids = sorted({op[1] for p in progs for op in p if op[0] in ("arrive", "sync")}) + ["meet"]
    start = ((0,) * len(progs), 0, (frozenset(),) * len(ids))
    seen, todo = {start}, [start]
    while todo:
        place, issued, arrived = todo.pop()
        moves = 0
        for a, prog in enumerate(progs):
            if place[a] == len(prog):
                continue
            op = prog[place[a]]
            new_place, new_issued, new_arrived = list(place), issued, list(arrived)
            if op[0] == "issue":
                new_issued += 1
                new_place[a] += 1
            elif op[0] == "group":
                if issued < op[1]:
                    continue
                new_place[a] += 1
            else:
                b = ids.index("meet" if op[0] == "meet" else op[1])
                waits = op[0] != "arrive"
                if a in arrived[b]:
                    if waits:
                        continue  # waiting there
                    return "double arrival"
                now = arrived[b] | {a}
                if not waits:
                    new_place[a] += 1
                # complete: as many arrivals as agents expected (all, or the compute warps among themselves)
                if len(now) == (COMPUTE if op[0] == "meet" else len(progs)):
                    for w in now:
                        at = progs[w][new_place[w]] if new_place[w] < len(progs[w]) else None
                        if at and at[0] in ("sync", "meet") and ids.index("meet" if at[0] == "meet" else at[1]) == b and (w == a or w in arrived[b]):
                            new_place[w] += 1
                    now = frozenset()
                new_arrived[b] = now
            moves += 1
            state = (tuple(new_place), new_issued, tuple(new_arrived))
            if state not in seen:
                seen.add(state)
                todo.append(state)
        if moves == 0 and any(place[a] < len(p) for a, p in enumerate(progs)):
            return "stuck"
    return "ok"


@pytest.mark.parametrize("units", [2, 4, 6])
@pytest.mark.parametrize("stop_after", [None, 0, 1, 2])
def test_handovers_never_meet(barriers, units, stop_after):
    assert explore(programs(lambda k: barriers[k], 3, units, stop_after)) == "ok"


def test_a_single_barrier_is_not_enough():
    assert explore(programs(lambda k: 5, 2, 2, None)) == "double arrival"
    assert explore(programs(lambda k: 5, 2, 2, 0)) == "double arrival"


def test_barriers_do_not_overlap_the_others(barriers):
    """1 to 4 are the gates' groups, 6 the compute warps' own, 0 the block's."""
    assert not set(barriers) & {0, 1, 2, 3, 4, 6} and max(barriers) < 16
