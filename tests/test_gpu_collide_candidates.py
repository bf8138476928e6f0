"""The collision tick's candidate tests (exact_ballpark_b200/csrc/ebb_collide.cu): the key ranges' meeting, the spheres' and
the statics' early refusals and the queue of reactions, against the oracle, bit for bit, where they can go wrong: balls in
and out of reach by a hair, at rest and fast, of no size and as wide as their boxes, few and many static collidables (more
than a world's slots and fewer), full and ragged blocks."""

import numpy as np
import pytest
import torch

import collide_trace as ct
from golden_util import bit_equal

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")]

FIELDS = ct.FIELDS


def _worlds(worlds: int, slots: int, statics: int, cube: float, seed: int) -> tuple:
    from exact_ballpark_b200.workloads import collide_statics_worlds, collide_worlds
    free = max(1, slots // 2)
    if statics:
        w = collide_statics_worlds(seed, worlds, free, slots - free, statics, ticks=1)
    else:
        w = collide_worlds(seed, worlds, free, 0, slots - free, ticks=1)
    g = np.random.default_rng(seed)
    for balls in w.worlds:
        for k, b in enumerate(balls):
            b["pos"] = (np.asarray(b["pos"]) * cube / 2e4).tolist()
            if b["free"] and k % 3 == 0:
                b["vel"] = [0.0, 0.0, 0.0]
            if k % 4 == 1:                               # touching the ball before it, or a millimetre off
                at = np.asarray(balls[k - 1]["pos"])
                gap = float(np.float32(b["radius"])) + float(np.float32(balls[k - 1]["radius"])) + g.choice([0.0, 1e-3, -1e-3])
                b["pos"] = (at + np.array([0.0, gap, 0.0])).tolist()
            if k % 5 == 2:
                b["radius"] = 0.0
    return w.worlds, w.collidables if statics else None


@pytest.mark.parametrize("worlds,slots,statics,cube", [(5, 1, 3, 2e4), (70, 2, 0, 500.0), (33, 16, 0, 2e4), (9, 17, 0, 3e3),
                                                       (7, 45, 0, 2e4), (3, 64, 0, 5e3), (41, 3, 1, 2e4), (21, 8, 8, 2e4),
                                                       (9, 8, 19, 2e4), (3, 40, 64, 2e4), (65, 2, 5, 4e3)])
def test_candidates_against_the_oracle(worlds, slots, statics, cube):
    from exact_ballpark_b200 import VecCollidePark
    from oracle.collide_park import OracleCollidePark
    balls, collidables = _worlds(worlds, slots, statics, cube, worlds + slots + statics)
    kw = {"statics": statics} if statics else {}
    a, b = OracleCollidePark(worlds, slots, **kw), VecCollidePark(worlds, slots, device="cuda", **kw)
    for p in (a, b):
        p.load(balls, collidables) if statics else p.load(balls)
    for k in range(8):
        a.evolve()
        b.evolve()
        for f in FIELDS:
            eq = bit_equal(np.asarray(getattr(a, f)), getattr(b, f).detach().cpu().numpy())
            assert eq.all(), (k, f, int((~eq).sum()))
