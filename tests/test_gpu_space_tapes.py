"""The size classes' tapes in one launch (ebb_space_tapes) on both sides of its line between few waves of blocks (more
registers) and many, against a thread a world (one launch a class, another kernel): every row, event count and flag."""

import numpy as np
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("worlds", [3, 10600, 10800])      # 2,664 blocks of 4 worlds: about 10,650 in six classes
def test_one_launch_of_the_classes_matches_a_thread_a_world(worlds):
    from exact_ballpark_b200.modes import VecModesPark, tick_tiled
    from exact_ballpark_b200.partition import CLASSES, PartitionLayer
    from exact_ballpark_b200.workloads import partition_worlds
    pw = partition_worlds(worlds, worlds)
    goto = torch.from_numpy(pw.cols["pos"] + np.random.default_rng(4).normal(0.0, 3e4, (pw.n, 3))).cuda()
    out = []
    for lanes, block in ((32, 128), (1, 64)):
        park = VecModesPark(pw.n, device="cuda")
        park.load_columns(pw.cols)
        part = PartitionLayer(park, pw.sizes, plan={c: (lanes, block) for c in CLASSES})
        part.load()
        part.add_sensors(pw.sensor_range, 1.0)
        park.goto_point(torch.ones(pw.n, dtype=torch.bool, device="cuda"), goto)
        for _ in range(3):
            part.tick(lambda park=park: tick_tiled(park))
            park.current_time += 1
        assert all(layer.lanes == lanes for layer, _ in part.layers)
        out.append([getattr(park, "_" + k).clone() for k in ("pos", "vel", "old_pos", "mode", "clock", "sensor", "radius")] +
                   [part.event_counts().clone(), part.flags().clone()])
        del park, part
    assert int(out[0][-2].sum()) > 0 and not (out[0][-1] != 0).any()
    assert all(torch.equal(a, b) for a, b in zip(*out))
