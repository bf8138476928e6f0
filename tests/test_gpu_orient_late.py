"""The torque searches of ships long in flight (exact_ballpark_b200/csrc/ebb_orient.cuh: a quarter of them are walked, from the
last candidate shown to fail) against the oracle's serial loops (oracle/flight.cpp), bit for bit over 200 ticks: few ships
a warp and full warps, short and long ticks."""

import numpy as np
import pytest
import torch

from golden_util import bit_equal

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")]

FIELDS = ("pos", "vel", "last_g", "rot", "old_rot", "ang_vel", "old_ang_vel", "torque", "rot_roll", "mode", "goto")


@pytest.mark.parametrize("worlds,tick_ms", [(6, 1000), (600, 1000), (600, 100)])
def test_a_long_flight_matches_the_serial_loops(worlds, tick_ms):
    from exact_ballpark_b200 import VecModesPark
    from exact_ballpark_b200.tiles import plan_tiles
    from exact_ballpark_b200.workloads import flight_worlds
    from oracle.park import OraclePark
    w = flight_worlds(worlds + tick_ms, worlds, 4)
    oracle, park = (c(len(w.rows), tick_interval_ms=tick_ms, dynamical_orientation=True, use_new_orbit=True)
                    for c in (OraclePark, VecModesPark))
    for p in (oracle, park):
        p.load(w.rows)
        w.apply(p)
    if worlds > 6:
        park.plan = plan_tiles(park.world, cap=256, block=256)        # full warps
    for k in range(1, 201):
        with np.errstate(all="ignore"):
            oracle.evolve()
        park.evolve()
        if k % 25:
            continue
        for f in FIELDS:
            eq = bit_equal(np.asarray(getattr(oracle, f)), getattr(park, f).detach().cpu().numpy())
            assert eq.all(), (k, f, int((~eq).sum()))
