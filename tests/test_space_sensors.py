"""The sensor checks' ahead-computed plan and its batches of 32 (exact_ballpark_b200/csrc/ebb_space.cuh), where they can go
wrong: ships around a corner where eight top boxes meet, so that a filing's boxes stay apart on every axis at every
level, and worlds whose sensors fill, miss by one, or pass a warp's batches. Every state and event of every tick
against the oracle's tick (oracle/space.cpp), bit for bit."""

import numpy as np
import pytest

import space_layer as sl
from oracle import space_world


def _worlds(ships: int, spread: float, seed: int):
    """A world of `ships` ships of the partition worlds' distributions, Gaussian around a corner of eight top boxes."""
    from exact_ballpark_b200.statics import LEVEL_WIDTH
    from exact_ballpark_b200.workloads import partition_worlds
    pw = partition_worlds(seed, 64)
    k = int(pw.starts[-1])
    g = np.random.default_rng(seed)
    pw.sizes = np.array([ships])
    for key in pw.cols:
        pw.cols[key] = np.resize(pw.cols[key], (max(ships, k),) + pw.cols[key].shape[1:])[:ships].copy()
    pw.cols["id"] = np.arange(1, ships + 1)
    pw.cols["pos"] = LEVEL_WIDTH[0] * np.array([1.0, -1.0, 2.0]) + g.normal(0.0, spread, (ships, 3))
    pw.sensor_range = 10.0 ** g.uniform(3.0, 5.4, ships)
    d = g.normal(0.0, 1.0, (ships, 3))
    return pw, pw.cols["pos"] + d / np.linalg.norm(d, axis=1, keepdims=True) * 1e9


def _differ(ships: int, spread: float, ticks: int, drive) -> list:
    bad = []
    for seed in (1, 2):
        pw, goto = _worlds(ships, spread, seed)
        ops = sl.partition_world_ops(pw, 0, goto, ticks)
        got = drive(ops, seed)
        want = [sl.oracle_lines(t, int(op[0])) for t, op in zip(space_world.run(ops, seed=seed), ops)]
        if got != want:
            bad.append((seed, next(i for i, (x, y) in enumerate(zip(want, got)) if x != y)))
    return bad


@pytest.mark.parametrize("ships,spread", [(1, 10.0), (2, 300.0), (7, 2e3), (24, 2e4), (40, 3e5)])
def test_plans_around_a_corner_of_eight_top_boxes(ships, spread):
    assert not _differ(ships, spread, 6, lambda ops, seed: sl.drive_ticks_host(ops, seed=seed))


@pytest.mark.gpu
@pytest.mark.parametrize("lanes,ships,spread", [(1, 4, 2e3), (32, 1, 10.0), (32, 4, 2e3), (32, 31, 1e4), (32, 32, 3e5),
                                                (32, 33, 2e3), (32, 65, 3e4), (32, 128, 1e5)])
def test_batches_of_sensors_on_the_device(lanes, ships, spread):
    import torch
    assert torch.cuda.is_available()
    assert not _differ(ships, spread, 4, lambda ops, seed: sl.drive_ticks(ops, seed=seed, lanes=lanes))


def test_several_layers_tapes_refuse_bad_arguments_before_launching():
    """ebb_space_tapes: too many layers, a thread-a-world or interleaved layer among them, a missing buffer; nothing to
    do without layers, worlds or operations."""
    import ctypes

    from exact_ballpark_b200 import _native
    lib = _native.lib()
    p = _native.FlightState()
    s, t = (_native.SpaceState * 2)(), (_native.SpaceTape * 2)()
    call = lambda n=2: lib.ebb_space_tapes(ctypes.byref(p), s, t, n, None)  # noqa: E731
    for k in range(2):
        for st in (p, s[k], t[k]):
            for name, kind in type(st)._fields_:
                if kind is ctypes.c_void_p:
                    setattr(st, name, 4096)
        s[k].worlds, s[k].slots, s[k].boxes, s[k].dicts, s[k].entries, s[k].sets = 0, 10, 64, 16, 16, 16
        s[k].umap_cap, s[k].events, s[k].lanes, s[k].pitch, t[k].K = 10, 16, 32, 1024, 1
    assert call(0) == 0 and call() == 0                   # no layers; no worlds
    assert call(-1) == -1 and call(_native.SPACE_MAX_LAYERS + 1) == -1
    s[1].worlds = 4
    for name, wrong in (("lanes", 1), ("pitch", 0), ("slots", 129), ("fbox", None), ("lanes", 7)):
        keep = getattr(s[1], name)
        setattr(s[1], name, wrong)
        assert call() == -1, name
        setattr(s[1], name, keep)
    t[1].code = None
    assert call() == -1
    t[1].K = 0
    assert call() == 0                                    # no operations
