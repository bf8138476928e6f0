"""The tile plan's autotuner (exact_ballpark_b200.autotune): the plan that a park was loaded with is timed among the
candidates, so that a tuned park is never slower by its own measurement than an untuned one, and the park's state is left
alone."""

import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("worlds,cands", [(64, None), (64, [(256, 256, None)]), (2000, None)])
def test_the_loaded_plan_is_a_candidate(worlds, cands):
    from exact_ballpark_b200 import VecModesPark
    from exact_ballpark_b200.autotune import autotune
    from exact_ballpark_b200.workloads import flight_worlds
    w = flight_worlds(3, worlds, 4)
    park = VecModesPark(len(w.rows), device="cuda", dynamical_orientation=True, use_new_orbit=True)
    park.load(w.rows)
    w.apply(park)
    loaded = (park.plan.cap, park.plan.block, park.plan.grid)
    before = {k: getattr(park, k).clone() for k in park.row_tensors()}
    times = autotune(park, cands=cands)
    assert loaded in times
    assert times[(park.plan.cap, park.plan.block, park.plan.grid)] == min(times.values()) <= times[loaded]
    for k, v in before.items():
        now = getattr(park, k)
        assert now.dtype == v.dtype and torch.equal(now.view(torch.uint8), v.view(torch.uint8)), k
