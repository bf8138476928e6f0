"""Re-filings at a ball's own level under its own top box (exact_ballpark_b200/csrc/ebb_space.cuh, refile_near), where they
can differ from leaving every box and entering again: sides coming, going and changing ends on each axis, boxes shared with
other balls or left empty with their ancestors, keys moved by one and by more, top boxes crossed now and then, and the
allocator's kept count from none to its 256, past the line from which the whole re-filing is taken. Every state after
every operation against the oracle's (oracle/space.cpp), bit for bit."""

import random

import numpy as np
import pytest

import space_layer as sl
import space_trace as sp
from exact_ballpark_b200.statics import LEVEL_WIDTH
from oracle import space_world

HUGE = 256                                                 # EBB_SPACE_FLAG_HUGE


def _stream(level: int, kept: int, seed: int):
    """Four balls filed at `level`, moved by up to 1.5 of its boxes around a corner of eight of them (the first axis one
    box from a top box's face), after `kept` balls far apart at the deepest level, added before them, were removed."""
    r = random.Random(f"refile-{level}-{kept}-{seed}")
    w = LEVEL_WIDTH[level]
    corner = [sp.TOP - w, 0.5 * sp.TOP, -0.25 * sp.TOP] if level else [sp.TOP, 0.0, -sp.TOP]
    add = lambda b, radius, x: sp._op(sp.ADD, b, 1e6, radius, 100.0, 1.0, 1.0, *x, 0.0, 0.0, 0.0, 1.0, 0.0, 1.0)  # noqa: E731
    where = lambda: [c + r.uniform(-1.5, 1.5) * w for c in corner]  # noqa: E731
    ops = [add(b, 20.0, [(3.3 + b % 4) * sp.TOP, (b // 4 + 0.3) * sp.TOP, 0.3 * sp.TOP]) for b in range(5, 5 + kept)]
    ops += [add(b, w * 0.3, where()) for b in range(1, 5)]
    ops += [sp._op(sp.REMOVE, b) for b in range(5, 5 + kept)]
    for _ in range(120):
        b = r.randint(1, 4)
        if r.random() < 0.05:
            ops.append(sp._op(sp.RADIUS, b, w * r.choice((0.01, 0.3, 0.33, 0.4))))
        else:
            ops.append(sp._op(sp.POS, b, *where()))
    return np.array(ops)


CASES = [(level, kept) for level in (0, 1, 4, 7) for kept in (0, 4, 12, 36)]


def _differ(where: str, **how) -> list:
    streams = [(_stream(level, kept, seed), 1) for level, kept in CASES for seed in (1, 2)]
    texts, flags = sl.drive(streams, where, **how)
    assert not (flags & ~HUGE).any()
    want = [[sl.oracle_lines(t, int(op[0])) for t, op in zip(space_world.run(ops, seed=s), ops)] for ops, s in streams]
    full = max(int(x.split()[1]) for ts in want for t in ts for x in t.splitlines() if x.startswith("F "))
    assert full >= 256                                    # (a chain begun below it is kept whole)
    return [(CASES[i // 2], next(k for k, (x, y) in enumerate(zip(b, a)) if x != y))
            for i, (a, b) in enumerate(zip(texts, want)) if a != b]


def test_refilings_near_by_on_the_cpu():
    assert not _differ("host")


@pytest.mark.gpu
@pytest.mark.parametrize("lanes", [1, 32])
def test_refilings_near_by_on_the_device(lanes):
    import torch
    assert torch.cuda.is_available()
    assert not _differ("cuda", lanes=lanes)
