"""Ticks whose dynamic shared memory alone fits the 48 KB that a block has by default, but not with the kernel's static arrays
beside it: one world of 479 to 483 ships (the tiled tick) or of 374 to 378 (the masked, listed-worlds tick) with the plan
that the park makes. In a process of its own, so that no earlier launch has opted in to more; each size asks for more than
the one before it. Held to the oracle bit for bit."""

import subprocess
import sys
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = """
import sys
sys.path[:0] = [{root!r}, {root!r} + "/tests"]
import numpy as np, torch
from exact_ballpark_b200 import VecModesPark
from exact_ballpark_b200.workloads import flight_worlds
from golden_util import bit_equal
from oracle.park import OraclePark
for ships in {sizes}:
    rows = []
    worlds = [flight_worlds(ships, 1, ships), flight_worlds(ships + 1, 1, 3)]
    for k, w in enumerate(worlds):
        rows += [dict(r, world=k) for r in w.rows]
    oracle, park = (c(len(rows), dynamical_orientation=True, use_new_orbit=True) for c in (OraclePark, VecModesPark))
    point = np.random.default_rng(ships).uniform(-1e5, 1e5, (len(rows), 3))
    oracle.load(rows)
    park.load(rows)
    oracle.goto_point(np.ones(len(rows), bool), point)
    park.goto_point(torch.ones(len(rows), dtype=torch.bool), torch.from_numpy(point))
    assert park.plan.cap == ships, park.plan.cap
    for _ in range(2):
        oracle.evolve()
        park.evolve(active=torch.ones(len(rows), dtype=torch.bool, device="cuda") if {masked} else None)
    torch.cuda.synchronize()
    for f in ("pos", "vel", "rot", "ang_vel", "torque", "clock"):
        assert bit_equal(np.asarray(getattr(oracle, f)), getattr(park, f).detach().cpu().numpy()).all(), (ships, f)
print("ticked")
"""


@pytest.mark.gpu
@pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")
@pytest.mark.parametrize("masked,sizes", [(False, [479, 480, 481, 482, 483]), (True, [374, 375, 376, 377, 378])])
def test_a_tick_whose_static_arrays_pass_the_default(masked, sizes):
    r = subprocess.run([sys.executable, "-c", PROGRAM.format(root=str(ROOT), sizes=sizes, masked=masked)], timeout=300,
                       capture_output=True, text=True)
    assert r.returncode == 0 and "ticked" in r.stdout, r.stdout + r.stderr
