"""The slot rule of the ring sweep (fp_ring_rule.h, compiled here with the host compiler) against the worst
order in which bulk copies can land: one position's copies are held back until nothing else can move.

The barriers are modelled as mbarriers are defined: a wait on parity P passes when the number of
completed phases is odd for P = 0 and even for P = 1.  Dependencies between elements only make a group
wait longer, so a schedule without any (the positions of finished cases) is the one to look at."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flowpro_v2_b200", "csrc")
SHIM = """#include "fp_ring_rule.h"
extern "C" int slots() { return fp::kRingSlots; }
extern "C" int may_request(int k, int tail, int inflight) { return fp::ring_may_request(k, tail, inflight); }
extern "C" unsigned parity(int k) { return fp::ring_lap_parity(k); }
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring")
    (d / "shim.cpp").write_text(SHIM)
    so = str(d / "shim.so")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", so, str(d / "shim.cpp")], check=True)
    return ctypes.CDLL(so)


def _passes(phases, parity):
    return phases % 2 != parity


def _run(rule, groups, late, total):
    """positions 0 .. total - 1, the copies of position `late` last; True when every position was
    multiplied with its own blocks"""
    n = rule.slots()
    full, empty = [0] * n, [0] * n  # completed phases
    head = tail = 0                 # requested, released (as the producer knows it)
    landed = set()
    at = list(range(groups))        # position each group waits on
    done = 0
    while done < total:
        moved = False
        while head < total and rule.may_request(head, tail, groups):
            if head != late:
                full[head % n] += 1
                landed.add(head)
            head += 1
            moved = True
        for g in range(groups):
            while at[g] < total and _passes(full[at[g] % n], rule.parity(at[g])):
                if at[g] not in landed:
                    return False  # another position's blocks
                empty[at[g] % n] += 1
                at[g] += groups
                done += 1
                moved = True
        while tail < head and _passes(empty[tail % n], rule.parity(tail)):
            tail += 1
            moved = True
        if not moved:
            if late in landed or late >= head:
                return False  # stuck for good
            full[late % n] += 1
            landed.add(late)
    return True


@pytest.mark.parametrize("groups", range(1, 17))
def test_no_group_takes_another_lap_for_its_own(rule, groups):
    n = rule.slots()
    for late in list(range(0, n + groups)) + [3 * n - 1, 3 * n]:
        assert _run(rule, groups, late, 5 * n + 7), (groups, late)
