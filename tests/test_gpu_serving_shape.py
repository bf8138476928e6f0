"""The serving loop's tile shape (exact_ballpark_b200.serving.Server): one that the caller names is the one that ticks, tiles of
many rows and several rounds of ships a block among them; without one it follows the live rows."""

import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a CUDA GPU")]


@pytest.mark.parametrize("named,cap,block", [({"tile_cap": 1024}, 1024, 256), ({"block": 64}, 256, 64),
                                             ({"tile_cap": 256, "block": 256}, 256, 256), ({"grid": 1}, 256, 256),
                                             ({"tile_cap": 96, "block": 32, "grid": 2}, 96, 32), ({}, None, None)])
def test_a_named_shape_is_kept(named, cap, block):
    from exact_ballpark_b200.serving import Server, episode_stream
    from exact_ballpark_b200.tiles import shape_for
    eps = episode_stream(5, 40, rate=0.0, max_ships=40, min_ships=2, min_ticks=12, max_ticks=12)
    with Server(rows=8192, max_ships=40, **named) as srv:
        for e in eps:
            srv.submit(e)
        steps = 0
        while steps < 4:
            ran = srv.step()
            if not ran:
                continue
            steps += 1
            assert len(srv.live) and srv._plan is not None
            want = (cap, block) if named else shape_for(srv.live_rows, int(srv.table.len[:srv.table.count].max()))
            assert tuple(srv._plan[3:]) == want
        srv.flush()
        srv.check()
