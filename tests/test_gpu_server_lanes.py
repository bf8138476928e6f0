"""Which lanes a server tick gives a world (exact_ballpark_b200/csrc/ebb_server.cu: lanes): many worlds a lane each, of more
rows than its registers hold too, against the same calls in a padded queue that takes a group of lanes, bit for bit; and
many worlds of one more ship cost no more than their share (a group of lanes for a longer queue cost four times as much)."""

import numpy as np
import pytest
import torch

from test_gpu_server_groups import _calls, _run

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")]


def same_bits(a, b) -> bool:
    """The same bits, or both NaN; integers and flags in their own type (no way through a double)."""
    if not a.dtype.is_floating_point:
        return torch.equal(a, b)
    bits = torch.int64 if a.dtype == torch.float64 else torch.int32
    return bool(((a.contiguous().view(bits) == b.contiguous().view(bits)) | (a.isnan() & b.isnan())).all())


def test_the_comparison_tells_bits_apart():
    one = torch.tensor([2 ** 62 + 1, 5])
    assert same_bits(one, one.clone()) and not same_bits(one, one - 1)
    z = torch.tensor([0.0, float("nan")])
    assert same_bits(z, z.clone()) and not same_bits(z, torch.tensor([-0.0, float("nan")]))
    assert not same_bits(z, torch.tensor([0.0, 0.0]))


@pytest.mark.parametrize("worlds,ships,shuffled,count", [(7000, 9, False, 4), (7000, 9, True, 4), (5000, 4, True, 11)])
def test_a_lane_a_world_matches_a_group(worlds, ships, shuffled, count):
    calls = _calls(worlds, ships, count, 11)
    want = _run(worlds, ships, shuffled, calls, [0] * (count + 1))
    pads = np.bincount(np.random.default_rng(5).integers(0, count + 1, 64), minlength=count + 1)
    got = _run(worlds, ships, shuffled, calls, pads.tolist())
    assert len(got) == len(want)
    for i, (a, b) in enumerate(zip(want, got)):
        assert a.dtype == b.dtype and same_bits(a, b), i


@pytest.mark.parametrize("worlds,ships,shuffled,count", [(37, 1, False, 3), (61, 4, True, 4), (19, 33, True, 9),
                                                         (11, 130, False, 12)])
def test_every_group_matches_by_bits(worlds, ships, shuffled, count):
    calls = _calls(worlds, ships, count, 3)               # (the calls' values hold NaN, -0.0 and warps' 64-bit patterns)
    want = _run(worlds, ships, shuffled, calls, [0] * (count + 1))
    for total in (8, 16, 33, 70):
        if total <= count:
            continue
        pads = np.bincount(np.random.default_rng(total).integers(0, count + 1, total - count), minlength=count + 1)
        got = _run(worlds, ships, shuffled, calls, pads.tolist())
        for i, (a, b) in enumerate(zip(want, got, strict=True)):
            assert a.dtype == b.dtype and same_bits(a, b), (total, i)


def test_a_longer_queue_costs_its_share():
    from exact_ballpark_b200 import VecModesPark, server
    us = []
    for ships in (4, 5):
        worlds = 65536
        n, g = worlds * ships, np.random.default_rng(ships)
        park = VecModesPark(n, device="cuda")
        park.load_columns({"id": np.tile(np.arange(1, ships + 1), worlds), "world": np.repeat(np.arange(worlds), ships),
                           "time": np.zeros(n, np.int64), "mass": np.full(n, 1e7), "radius": np.full(n, 50.0),
                           "max_vel": np.full(n, 200.0), "agility": np.ones(n), "speed_fraction": np.ones(n),
                           "free": np.ones(n, bool), "massive": np.zeros(n, bool), "interactive": np.ones(n, bool),
                           "moribund": np.zeros(n, bool), "cloaked": np.zeros(n, np.int64),
                           "bubble": np.zeros(n, np.int64), "mode": np.full(n, 2, np.int64), "max_ang_vel": np.ones(n),
                           "rot_agility": np.full(n, 0.9), "pos": g.uniform(-4e3, 4e3, (n, 3)), "vel": np.zeros((n, 3))})
        srv = server.VecServer(server.ModesAdapter(park), list(range(ships)) * worlds, kernel="cuda")
        srv.pre_tick()
        srv.evolve()
        srv.post_tick()
        graph = server.ServerGraph(srv, ["GotoDirection", "SetSpeedFraction"] * ships)
        for k, x in enumerate(graph.inputs):
            x["mask"].fill_(True)
            x["ball"].fill_(k // 2 + 1)
            x["f"].fill_(0.5)
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            graph.tick()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b) * 1e3)
        us.append(min(times))
    assert us[1] < 2.5 * us[0], us                       # 1.25 times its rows and calls; a group a world: 4.2 times
