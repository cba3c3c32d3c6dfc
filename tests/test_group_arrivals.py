"""How the small groups' products meet (step_group.cu), restated: at each pair of the
tree the first group to arrive ends and the second goes on.  Whatever launches that
overlapped on one context left in the arrival numbers, a launch by itself takes every
pair exactly once and never before both of its groups have come, in any order of the
groups; and a graph's replays too, which have one turn and clear the numbers first.
"""
import os
import random

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "parament_gb300", "csrc")


def group(chunk, n, arrived, turn, takes):
    """A group's walk up the tree; yields before every access to the numbers."""
    first = chunk
    level = 0
    while (1 << level) < n:
        right = (first >> level) & 1
        lo = first - (1 << level) if right else first
        hi = lo + (1 << level)
        if hi < n:
            yield
            before, arrived[hi] = arrived[hi], turn
            if before != turn:
                return
            yield
            arrived[hi] = 0
            takes.append((lo, hi, level))
            first = lo
        level += 1
    takes.append("root")


def launch(rng, n, arrived, turns):
    """One or more launches (by their turns) whose groups' accesses interleave."""
    takes = [[] for _ in turns]
    live = [group(c, n, arrived, t, k) for t, k in zip(turns, takes) for c in range(n)]
    while live:
        g = rng.randrange(len(live))
        try:
            next(live[g])
        except StopIteration:
            live.pop(g)
    return takes


def pairs(n):
    out, level = ["root"], 0
    while (1 << level) < n:
        out += [(lo, lo + (1 << level), level) for lo in range(0, n, 2 << level) if lo + (1 << level) < n]
        level += 1
    return sorted(out, key=str)


@pytest.mark.parametrize("n", [1, 2, 3, 7, 16, 29, 64])
def test_a_launch_takes_every_pair_once(n):
    rng = random.Random(n)
    for _ in range(200):
        arrived, turn = [0] * n, 0
        for kind in rng.choices(("alone", "overlapping"), k=6):
            if kind == "overlapping":  # their results are nobody's concern
                launch(rng, n, arrived, [turn + 1, turn + 2])
                turn += 2
            else:
                turn += 1
                takes, = launch(rng, n, arrived, [turn])
                assert sorted(takes, key=str) == pairs(n)
                done = set()
                for lo, hi, level in takes[:-1]:  # both halves were complete
                    for node, l in ((lo, level - 1), (hi, level - 1)):
                        if l >= 0 and node + (1 << l) < n:
                            assert (node, l) in done
                    done.add((lo, level))
                    done |= {(lo, k) for k in range(level)}


def test_replays_clear_the_numbers(n=13):
    rng = random.Random(5)
    arrived = [0] * n
    for _ in range(100):
        if rng.random() < 0.5:
            launch(rng, n, arrived, [7, 7])  # two replays at once
        arrived[:] = [0] * n
        takes, = launch(rng, n, arrived, [7])
        assert sorted(takes, key=str) == pairs(n)


def test_the_kernel_uses_turns():
    src = open(os.path.join(CSRC, "step_group.cu")).read()
    assert "atomicExch(&a.arrived[hi], a.turn) == a.turn" in src and "if (second) a.arrived[hi] = 0;" in src
