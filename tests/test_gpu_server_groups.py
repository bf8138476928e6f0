"""The server kernel's lanes a world (exact_ballpark_b200/csrc/ebb_server.cu): the same calls as a queue of 4, 8, 16, 32 or
more slots (padding pushes that no world makes, before, between and after them) leave the same park, flags, routes and
sends (8,300 worlds are taken a lane a world, and with padding a group a world). The narrow queues are held to the reference by the golden ticks (test_gpu_server.py); here every kind the park
takes meets a queue taken in several rounds, duplicates across a round's edge, and worlds of more rows than lanes, their
ids in order and not."""

import numpy as np
import pytest


def _server(worlds: int, ships: int, shuffled: bool, seed: int):
    from exact_ballpark_b200 import VecModesPark, server
    g = np.random.default_rng(seed)
    rows = []
    for w in range(worlds):
        ids = np.arange(1, ships + 1)
        if shuffled:
            g.shuffle(ids)
        for i in ids:
            rows.append({"id": int(i), "world": w, "time": 0, "mass": 10 ** g.uniform(6, 8), "radius": g.uniform(20, 80),
                         "max_vel": g.uniform(100, 400), "pos": g.uniform(-4e3, 4e3, 3).tolist(),
                         "vel": g.uniform(-50, 50, 3).tolist(), "agility": g.uniform(0.3, 1.5), "speed_fraction": 1.0,
                         "interactive": bool(g.random() < 0.8), "bubble": 0})
    park = VecModesPark(len(rows), device="cuda", dynamical_orientation=True)
    park.load(rows)
    return server.VecServer(server.ModesAdapter(park), [k if g.random() < 0.9 else -1 for k in range(len(rows))])


def _calls(worlds: int, ships: int, count: int, seed: int) -> list:
    """`count` pushes of random kinds and arguments (the values few, so that calls repeat), each masked to some worlds."""
    from exact_ballpark_b200 import server
    import torch
    g = np.random.default_rng(seed)
    takes = [k for k in range(1, len(server.KINDS)) if server.KINDS[k] not in ("LaunchMissile", "AddBallsToPark",
                                                                              "BallNotGlobal")]
    out = []
    for j in range(count):
        if j and g.random() < 0.35:                       # the call before again, in some worlds with another argument
            k, mask, ball, target, f, n = out[-1]
            f = f.clone()
            f[torch.from_numpy(g.random(worlds) < 0.3)] = 0.5
        else:
            k = int(g.choice(takes))
            ball = torch.from_numpy(g.integers(0, min(ships, 5) + 2, worlds))
            target = torch.from_numpy(g.integers(1, ships + 1, worlds))
            f = torch.from_numpy(g.choice([0.0, -0.0, 1.0, 0.5, 700.0, 3e5, float("nan")], (worlds, 4)))
            n = torch.from_numpy(g.integers(0, 3, worlds))
        out.append((k, torch.from_numpy(g.random(worlds) < 0.8), ball, target, f, n))
    return out


def _run(worlds: int, ships: int, shuffled: bool, calls: list, pads: list) -> list:
    import torch
    s = _server(worlds, ships, shuffled, 7)
    s.tick()
    none = torch.zeros(worlds, dtype=torch.bool)
    out = []
    for t in range(2):
        slots = []
        for j, (k, mask, ball, target, f, n) in enumerate(calls):
            for _ in range(pads[j]):
                s.push("GotoPoint", none, ball)
            slots.append(s.push(k, mask, ball, target, f, n))
        for _ in range(pads[-1]):
            s.push("CloakBall", none, calls[0][2])
        s.pre_tick(snapshot=False)
        at = [k for k, x in enumerate(s.batch.slots) if any(x is y for y in slots)]
        assert len(at) == len(calls)
        out += [s.batch.route[:, at].clone()] + [x.clone() for y in slots for x in (y.ok, y.row, y.trow, y.loc)]
        out += [rec.clone() for j, rec, _ in s.batch.notices]
        s.evolve()
        s.post_tick()
        out += [s.batch.has_character.clone(), s.batch.gets_bubble.clone(), s.dead.clone()]
    p = s.a.park
    return out + [getattr(p, k).clone() for k in p.row_tensors()] + [p.cloaked.clone(), p.bubble.clone()]


@pytest.mark.gpu
@pytest.mark.parametrize("worlds,ships,shuffled,count", [(37, 1, False, 3), (61, 4, True, 4), (33, 5, False, 7),
                                                         (19, 33, True, 9), (11, 130, False, 12),
                                                         (8300, 3, True, 4)])
def test_a_queues_padding_changes_nothing(worlds, ships, shuffled, count):
    import torch
    assert torch.cuda.is_available()
    for seed in (1, 2, 3) if worlds < 1000 else (4,):
        calls = _calls(worlds, ships, count, seed)
        want = _run(worlds, ships, shuffled, calls, [0] * (count + 1))
        g = np.random.default_rng(seed)
        for total in (8, 16, 32, 33, 70):
            if total <= count:
                continue
            pads = np.bincount(g.integers(0, count + 1, total - count), minlength=count + 1)
            got = _run(worlds, ships, shuffled, calls, pads.tolist())
            assert len(got) == len(want)
            for i, (a, b) in enumerate(zip(want, got)):
                assert torch.equal(torch.nan_to_num(a.double()), torch.nan_to_num(b.double())), (seed, total, i)
