"""The rules of the lane loop that need no GPU (csrc/dms_lane_rules.h), compiled for the host."""
import ctypes
import os
import subprocess

import pytest

from dms_ctypes import PACKAGE_DIR, REPO

SHIM = r"""
#include "dms_lane_rules.h"
extern "C" {
int vote_sets() { return dms::lane::VOTE_SETS; }
int next_vote_set(int set) { return dms::lane::next_vote_set(set); }
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text(SHIM)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(PACKAGE_DIR, "csrc"),
                    "-I", os.path.join(REPO, "include"), "-o", str(d / "rules.so"), str(d / "rules.cpp")], check=True)
    return ctypes.CDLL(str(d / "rules.so"))


def wrong_count_possible(warps, passes, sets, following, clear_after_barrier):
    """Whether some order of the warps' accesses gives a warp a wrong count.

    In each pass every warp adds 1 to the pass's set, waits for the others and reads the set; warp 0 also clears
    the set of the next pass, before the barrier or after its read.  All orders that the barrier allows are tried."""
    body = ["add", "wait", "read"]
    first = body + ["clear"] if clear_after_barrier else ["clear"] + body
    programs = [[(op, p) for p in range(passes) for op in (first if w == 0 else body)] for w in range(warps)]
    set_of = [0]
    for _ in range(passes):
        set_of.append(following(set_of[-1]))

    def passed(w, at):
        """Barriers that a warp at this position is past."""
        return sum(op == "wait" for op, _ in programs[w][:at])

    seen, todo = set(), [((0,) * warps, (0,) * sets)]  # positions, counts
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        at, counts = state
        for w in range(warps):
            if at[w] == len(programs[w]):
                continue
            op, p = programs[w][at[w]]
            # a barrier opens when every warp has reached it
            if op == "wait" and not all(passed(u, at[u]) > p or programs[u][at[u]] == ("wait", p) for u in range(warps)):
                continue
            if op == "read" and counts[set_of[p]] != warps:
                return True
            c = list(counts)
            if op == "add":
                c[set_of[p]] += 1
            elif op == "clear":
                c[set_of[p + 1]] = 0
            todo.append((at[:w] + (at[w] + 1,) + at[w + 1:], tuple(c)))
    return False


@pytest.mark.parametrize("warps", [2, 3])
def test_no_vote_of_a_block_in_lockstep_is_lost(rules, warps):
    assert not wrong_count_possible(warps, 5, rules.vote_sets(), rules.next_vote_set, clear_after_barrier=False)


def test_two_vote_sets_are_too_few():
    """The search finds the races that it is made for."""
    def other(s):
        return 1 - s
    assert wrong_count_possible(2, 3, 2, other, clear_after_barrier=True)
    assert wrong_count_possible(2, 3, 2, other, clear_after_barrier=False)
