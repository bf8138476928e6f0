"""The torque searches' guess, bounds and walk (exact_ballpark_b200/csrc/ebb_orient.cuh) against the oracle's serial loops
(oracle/flight.cpp), bit for bit, where they can go wrong: ships whose turning takes one candidate or all 99, kappas that
vanish or stay at one, turning rates far past the maximum and far below it, zero and huge maxima (outside the bounds'
ranges), short and long ticks, and warps of few ships."""

import numpy as np
import pytest
import torch

from golden_util import bit_equal

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")]

FIELDS = ("pos", "vel", "last_g", "rot", "old_rot", "ang_vel", "old_ang_vel", "torque", "rot_roll", "mode")


def _pair(n: int, seed: int, tick_ms: int, wide: bool):
    from exact_ballpark_b200 import VecModesPark
    from oracle.park import OraclePark
    g = np.random.default_rng(seed)
    lo, hi = (0.0, 13.0) if wide else (4.0, 10.0)
    rows = [{"id": i % 8 + 1, "world": i // 8, "time": 0, "mass": 10 ** g.uniform(lo, hi), "radius": g.uniform(20, 500),
             "max_vel": 10 ** g.uniform(2, 3.5), "pos": g.uniform(-5e4, 5e4, 3).tolist(),
             "vel": g.uniform(-300, 300, 3).tolist(), "agility": g.uniform(0.01, 5), "speed_fraction": 1.0,
             "max_ang_vel": 10 ** (g.uniform(-12, 9) if wide else g.uniform(-3, 1)),
             "rot_agility": 10 ** (g.uniform(-4, 4) if wide else g.uniform(-1, 1))} for i in range(n)]
    parks = (OraclePark(n, tick_interval_ms=tick_ms, dynamical_orientation=True, use_new_orbit=True),
             VecModesPark(n, tick_interval_ms=tick_ms, dynamical_orientation=True, use_new_orbit=True))
    cmd = g.integers(0, 3, n)
    target = np.arange(n) // 8 * 8 + (np.arange(n) + g.integers(1, 8, n)) % 8
    rng, point = g.uniform(500, 3e4, n), g.uniform(-1e5, 1e5, (n, 3))
    spin = g.normal(0, 1, (n, 3)) * (10 ** g.uniform(-6, 3, n))[:, None]
    still = g.random(n) < 0.5
    quat = g.normal(0, 1, (n, 4))
    for p in parks:
        t = (lambda a: a) if isinstance(p, OraclePark) else (lambda a: torch.from_numpy(np.ascontiguousarray(a)))
        p.load(rows)
        p.follow(t(cmd == 0), t(target), t(rng))
        p.orbit(t(cmd == 1), t(target), t(rng))
        p.goto_point(t(cmd == 2), t(point))
        p.set_rotation(t(~still), t(quat))
        p.set_angular_velocity(t(~still), t(spin))
    return parks


@pytest.mark.parametrize("tick_ms", [50, 1000, 20000])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("n", [8, 24, 4096])
def test_the_searches_match_the_serial_loops(n, wide, tick_ms):
    oracle, park = _pair(n, n + tick_ms + wide, tick_ms, wide)
    for k in range(12):
        with np.errstate(all="ignore"):
            oracle.evolve()
        park.evolve()
        for f in FIELDS:
            eq = bit_equal(np.asarray(getattr(oracle, f)), getattr(park, f).detach().cpu().numpy())
            assert eq.all(), (k, f, int((~eq).sum()))
