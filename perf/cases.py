"""The work that users of this framework run, as cases to measure: one pass a case through the public entry points.

Every park is a simulator that a program steps many times, so a pass is a rollout: the park's state set back to the
case's start (its tensors copied from a snapshot on the device, as a planner or a learner resets its worlds), the
pilots' commands where the case has them, then `ticks` ticks through the graph wrappers, `evolve` or the serving loop.
Every pass of a state is therefore the same work on the same worlds, however often it is repeated. The outputs are the
parks' state after the last tick, with the collision lists, the events and the filings that the ticks write.

`listed()` names the cases, `draw(rng)` gives further ones of the same ranges, `prepare(case, seed)` makes the worlds
from the seed (numpy draws of the distributions of exact_ballpark_b200.workloads) and loads them, `run(state)` is one
pass, `work(case)` the bytes and operations that its ticks cannot do without, `exact(case, seed)` the pilots' flights in
64-bit arithmetic without this package's code (the other ticks have no value but the bit-exact one: they round to
floats at fixed places, branch on the results and answer collisions in a fixed order).
"""

import math

import numpy as np
import torch

from exact_ballpark_b200 import CollideGraph, CombatGraph, ModesGraph, VecCollidePark, VecCombatPark, VecComposedPark
from exact_ballpark_b200 import VecModesPark, server
from exact_ballpark_b200.partition import partition_setup
from exact_ballpark_b200.serving import Episode, Server, serve
from exact_ballpark_b200.workloads import (COMBAT_FORMATIONS, CombatWorlds, PackedWorlds, PartitionWorlds,
                                           collide_statics_worlds, collide_worlds, face_worlds, flight_worlds)

TEMPLATES = 512          # collision worlds drawn and loaded one by one; a larger park holds them several times over


def listed() -> list:
    return [
        # the smallest batch: one scenario's 64 worlds of 4 ships stepped for 200 game seconds; launches and latency
        {"name": "flight_64x4", "kind": "flight", "worlds": 64, "ships": 4, "ragged": False, "orientation": True,
         "new_orbit": True, "masked": False, "ticks": 200},
        # the flight benchmark's batch: a learner's or a simulator farm's wide batch of small worlds
        {"name": "flight_65536x4", "kind": "flight", "worlds": 65536, "ships": 4, "ragged": False,
         "orientation": True, "new_orbit": True, "masked": False, "ticks": 8},
        # worlds of uneven size, an odd number of them, some held back by OnTick's mask every tick, the older orbit
        {"name": "flight_ragged_masked", "kind": "flight", "worlds": 2999, "ships": 128, "ragged": True,
         "orientation": True, "new_orbit": False, "masked": True, "ticks": 8},
        # continuous batching: episodes of 1 to 256 ships submitted together, staged, admitted, ticked to their ends
        {"name": "serve_256", "kind": "serve", "episodes": 256, "ships": 256, "min_ticks": 10, "ticks": 100},
        # ships flying into free and fixed spheres: the gradient method
        {"name": "collide_16384x16", "kind": "collide", "worlds": 16384, "ships": 4, "free": 4, "fixed": 8,
         "statics": 0, "ticks": 10},
        # crowded worlds of an odd size, near the largest the park takes
        {"name": "collide_1023x45", "kind": "collide", "worlds": 1023, "ships": 15, "free": 15, "fixed": 15,
         "statics": 0, "ticks": 10},
        # stations and asteroids: capsules and oriented boxes beside the balls
        {"name": "statics_16384x8+8", "kind": "collide", "worlds": 16384, "ships": 4, "free": 0, "fixed": 4,
         "statics": 8, "ticks": 10},
        # missiles and formations
        {"name": "combat_16384x8", "kind": "combat", "worlds": 16384, "ships": 4, "missiles": 4, "spheres": 0,
         "ticks": 8},
        # missiles, formations and collisions in one park
        {"name": "composed_16384x9", "kind": "composed", "worlds": 16384, "ships": 6, "missiles": 2, "spheres": 1,
         "ticks": 8},
        # the server layer: every ship piloted, two calls a ship a tick
        {"name": "server_65536x4", "kind": "server", "worlds": 65536, "ships": 4, "ticks": 16},
        # the ragged batch with bubbles, the partition, proximity sensors and the server on top
        {"name": "partition_8000x128", "kind": "partition", "worlds": 8000, "ships": 128, "ticks": 4},
        # small worlds across a top box's face: every ship re-files every tick, bubbles and sensors change
        {"name": "face_16384x4", "kind": "face", "worlds": 16384, "ships": 4, "ticks": 4},
    ]


def _log(rng, lo: int, hi: int) -> int:
    """A whole number of [lo, hi], uniform in its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng) -> dict:
    """One more case: any kind, its sizes over the range up to the listed ones', odd ones among them."""
    kind = rng.choice(("flight", "flight", "serve", "collide", "collide", "collide", "combat", "composed", "server",
                       "partition", "face"))
    ticks = rng.randint(4, 8)
    if kind == "flight":
        ragged = rng.random() < 0.5
        return {"kind": kind, "worlds": _log(rng, 64, 2999) if ragged else _log(rng, 64, 65536),
                "ships": rng.randint(8, 128) if ragged else rng.randint(2, 4), "ragged": ragged,
                "orientation": rng.random() < 0.75, "new_orbit": rng.random() < 0.5, "masked": rng.random() < 0.4,
                "ticks": ticks}
    if kind == "serve":
        return {"kind": kind, "episodes": _log(rng, 16, 256), "ships": rng.randint(16, 256), "min_ticks": 10,
                "ticks": rng.randint(20, 100)}
    if kind == "collide":
        if rng.random() < 0.4:
            return {"kind": kind, "worlds": _log(rng, 64, 16384), "ships": rng.randint(1, 4), "free": 0,
                    "fixed": rng.randint(1, 4), "statics": rng.randint(1, 8), "ticks": ticks}
        if rng.random() < 0.5:
            return {"kind": kind, "worlds": _log(rng, 64, 1023), "ships": rng.randint(3, 15),
                    "free": rng.randint(3, 15), "fixed": rng.randint(3, 15), "statics": 0, "ticks": ticks}
        return {"kind": kind, "worlds": _log(rng, 64, 16384), "ships": rng.randint(1, 4), "free": rng.randint(1, 4),
                "fixed": rng.randint(0, 8), "statics": 0, "ticks": ticks}
    if kind == "combat":
        return {"kind": kind, "worlds": _log(rng, 64, 16384), "ships": rng.randint(2, 4),
                "missiles": rng.randint(1, 4), "spheres": 0, "ticks": ticks}
    if kind == "composed":
        return {"kind": kind, "worlds": _log(rng, 64, 16384), "ships": rng.randint(2, 6),
                "missiles": rng.randint(1, 2), "spheres": rng.randint(0, 1), "ticks": ticks}
    if kind == "server":
        return {"kind": kind, "worlds": _log(rng, 64, 65536), "ships": rng.randint(1, 4), "ticks": 2 * ticks}
    if kind == "partition":
        return {"kind": kind, "worlds": _log(rng, 64, 8000), "ships": rng.choice((16, 32, 64, 100, 128)),
                "ticks": 4}
    return {"kind": kind, "worlds": _log(rng, 64, 16384), "ships": 4, "ticks": 4}


# ============================================================================ the worlds

def _unit(g, n: int) -> np.ndarray:
    d = g.normal(0.0, 1.0, (n, 3))
    return d / np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-9)


def _ship_columns(g, sizes: np.ndarray) -> dict:
    """Load columns of worlds of `sizes` ships, ids from 1 in each: the flight benchmark's distributions."""
    n = int(sizes.sum())
    starts = np.concatenate(([0], np.cumsum(sizes)[:-1]))
    return {"id": np.arange(n) - np.repeat(starts, sizes) + 1, "world": np.repeat(np.arange(len(sizes)), sizes),
            "time": np.zeros(n, np.int64), "mass": 10.0 ** g.uniform(6.0, 9.0, n), "radius": g.uniform(20.0, 500.0, n),
            "max_vel": 10.0 ** g.uniform(2.0, math.log10(3000.0), n), "agility": g.uniform(0.1, 5.0, n),
            "speed_fraction": np.ones(n), "free": np.ones(n, bool), "massive": np.zeros(n, bool),
            "interactive": g.random(n) < 0.5, "moribund": np.zeros(n, bool), "cloaked": np.zeros(n, np.int64),
            "bubble": np.full(n, -1, np.int64), "mode": np.full(n, 2, np.int64), "max_ang_vel": np.ones(n),
            "rot_agility": np.full(n, 0.9), "pos": g.uniform(-5e4, 5e4, (n, 3)), "vel": np.zeros((n, 3))}


def _others(g, sizes: np.ndarray) -> np.ndarray:
    """Each row's uniform other row of its world (its own in a world of one)."""
    starts = np.repeat(np.concatenate(([0], np.cumsum(sizes)[:-1])), sizes)
    size = np.repeat(sizes, sizes)
    me = np.arange(int(sizes.sum())) - starts
    step = 1 + np.floor(g.random(len(me)) * np.maximum(size - 1, 1)).astype(np.int64)
    return starts + np.where(size > 1, (me + step) % size, me)


def _ragged(count: int, most: int) -> np.ndarray:
    """Ship counts log-uniform in [1, most]; of the case alone, so that every seed's batch has the same rows."""
    g = np.random.default_rng([count, most])
    return np.clip(np.floor(10.0 ** g.uniform(0.0, math.log10(most), count)), 1, most).astype(np.int64)


def _flight_worlds(g, sizes: np.ndarray) -> PackedWorlds:
    """Each ship FOLLOW or ORBIT of another ship of its world, or WARP (always in a world of one ship)."""
    cols = _ship_columns(g, sizes)
    n = len(cols["id"])
    mode = np.where(np.repeat(sizes, sizes) > 1, g.integers(0, 3, n), 2)
    point = cols["pos"] + _unit(g, n) * (10.0 ** g.uniform(8.0, 11.0, n))[:, None]
    return PackedWorlds(cols, mode == 0, mode == 1, mode == 2, np.where(mode < 2, _others(g, sizes), -1),
                        np.where(mode < 2, g.uniform(500.0, 30000.0, n), 0.0), np.where((mode == 2)[:, None], point, 0.0),
                        np.where(mode == 2, g.integers(3000, 10001, n), 0), len(sizes))


def _rows(cols: dict, **more) -> list:
    """Columns as the list of row dicts that a park's load takes."""
    cols = {**cols, **more}
    keys = list(cols)
    return [dict(zip(keys, v)) for v in zip(*(c.tolist() if isinstance(c, np.ndarray) else c for c in cols.values()))]


def _combat_worlds(g, case: dict) -> CombatWorlds:
    """Worlds of ships, fixed spheres and missiles in the shape of workloads.combat_worlds and composed_worlds."""
    W, S, Q, M = case["worlds"], case["ships"], case["spheres"], case["missiles"]
    composed = case["kind"] == "composed"
    cube = 5e3 if composed else 2e4
    per, n = S + Q + M, W * (S + Q + M)
    j = np.tile(np.arange(per), W)
    base = np.repeat(np.arange(W) * per, per)
    ship, sphere, missile = j < S, (j >= S) & (j < S + Q), j >= S + Q
    u = lambda lo, hi: g.uniform(lo, hi, n)
    pick = lambda a, b, c: np.where(ship, a, np.where(sphere, b, c))
    pos = np.where(missile[:, None], 0.0, g.uniform(-cube, cube, (n, 3)))
    still = np.zeros((n, 3))
    rows = _rows({"id": np.where(missile, 101 + j - S - Q, j + 1), "world": np.repeat(np.arange(W), per),
                  "time": np.zeros(n, np.int64), "exists": ~missile, "mass": pick(10.0 ** u(6, 9), 10.0 ** u(8, 11), 1.0),
                  "radius": pick(u(20, 500), 10.0 ** u(1.0, math.log10(5000.0)), 1.0),
                  "max_vel": pick(10.0 ** u(2.0, math.log10(3000.0)), 0.0, 1.0), "pos": pos, "vel": still,
                  "agility": np.where(ship, u(0.1, 5.0), 1.0), "speed_fraction": np.where(sphere, 0.0, 1.0),
                  "free": ~sphere, "massive": sphere | (ship & composed),
                  "interactive": ship & ((j == 0) | (g.random(n) < 0.5))})
    mode = np.where(ship, g.integers(0, 3, n) if S > 1 else 2, -1)
    step = 1 + np.floor(g.random(n) * max(S - 1, 1)).astype(np.int64)
    other = (j + step) % S
    member = np.zeros(n, bool)
    leader = np.zeros(n, bool)
    formation, slot = np.zeros(n, np.int64), np.zeros(n, np.int64)
    if S > 1:                                    # in half the worlds ship 1 leads a formation, ship 2 flies in a slot
        lead = np.nonzero(g.random(W) < 0.5)[0] * per
        leader[lead] = True
        formation[lead] = g.integers(0, len(COMBAT_FORMATIONS), len(lead))
        member[lead + 1] = True
        slots = np.array([len(f) for f in COMBAT_FORMATIONS])[formation[lead]]
        slot[lead + 1] = np.floor(g.random(len(lead)) * slots).astype(np.int64)
    k = np.nonzero(missile)[0]
    m = len(k)
    owner = g.integers(0, S, m)
    target = (owner + 1 + np.floor(g.random(m) * max(S - 1, 1)).astype(np.int64)) % S
    balls = _rows({"id": 101 + j[k] - S - Q, "mass": 10.0 ** g.uniform(3, 5, m), "radius": g.uniform(1, 6, m),
                   "max_vel": g.uniform(3000, 8000, m), "free": np.ones(m, bool), "massive": np.zeros(m, bool),
                   "interactive": np.zeros(m, bool), "pos": np.zeros((m, 3)), "vel": np.zeros((m, 3)),
                   "agility": g.uniform(0.01, 0.2, m), "speed_fraction": np.ones(m),
                   "max_ang_vel": g.uniform(0.5, 3.0, m), "rot_agility": g.uniform(0.2, 1.0, m)})
    launch_target, launch_owner = np.zeros(n, np.int64), np.zeros(n, np.int64)
    launch_target[k], launch_owner[k] = target + 1, owner + 1
    return CombatWorlds(rows, W, S, M, mode == 0, mode == 1, mode == 2, np.where((mode == 0) | (mode == 1), base + other, -1),
                        np.where((mode == 0) | (mode == 1), u(500.0, 30000.0), 0.0),
                        np.where((mode == 2)[:, None], g.uniform(-cube, cube, (n, 3)), 0.0), leader, formation, member,
                        np.where(member, 1, 0), slot, missile, balls, launch_target, launch_owner)


def _server_worlds(g, worlds: int, ships: int) -> dict:
    """The server benchmark's worlds: ships near a centre, at rest, interactive, each with its pilot's two calls."""
    sizes = np.full(worlds, ships)
    cols = _ship_columns(g, sizes)
    n = worlds * ships
    cols.update(mass=10.0 ** g.uniform(6.0, 8.0, n), radius=g.uniform(20.0, 80.0, n), max_vel=g.uniform(100.0, 400.0, n),
                agility=g.uniform(0.3, 1.5, n), interactive=np.ones(n, bool), bubble=np.zeros(n, np.int64),
                pos=np.repeat(g.uniform(-1e5, 1e5, (worlds, 3)), ships, axis=0) + g.uniform(-4e3, 4e3, (n, 3)))
    return {"cols": cols, "direction": g.uniform(-1.0, 1.0, (n, 3)), "speed": g.uniform(0.0, 1.0, n)}


def _partition_worlds(case: dict, seed: int) -> PartitionWorlds:
    if case["kind"] == "face":
        return face_worlds(seed, case["worlds"])
    sizes = _ragged(case["worlds"], case["ships"])
    g = np.random.default_rng(seed)
    cols = _ship_columns(g, sizes)               # as workloads.partition_worlds draws them, the sizes apart
    n, world = len(cols["id"]), cols["world"]
    pick = (g.random(n) * g.integers(1, 6, len(sizes))[world]).astype(np.int64)
    cols["pos"] = g.uniform(-1e6, 1e6, (len(sizes), 5, 3))[world, pick] + g.normal(0.0, 1e4, (n, 3))
    cols["interactive"] = np.ones(n, bool)
    return PartitionWorlds(cols, sizes, 10.0 ** g.uniform(3.0, math.log10(2.5e5), n), _unit(g, n), g.uniform(0.2, 1.0, n))


# ============================================================================ preparing and running

class Snapshot:
    """Copies of a program's tensors on the device, and the copy back that starts a rollout."""

    def __init__(self, tensors: list):
        buffers = {}
        for t in tensors:                        # each tensor's whole buffer once (several are views of one)
            s = t.untyped_storage()
            if s.nbytes():
                buffers[s.data_ptr()] = torch.empty(0, dtype=torch.uint8, device=t.device).set_(s)
        self.live = list(buffers.values())
        self.kept = [b.clone() for b in self.live]
        small = [b.numel() < 1 << 20 for b in self.live]
        self.small = [[b for b, s in zip(bs, small) if s] for bs in (self.live, self.kept)]
        self.large = [(a, b) for a, b, s in zip(self.live, self.kept, small) if not s]

    def restore(self) -> None:
        if self.small[0]:
            torch._foreach_copy_(self.small[0], self.small[1])
        for a, b in self.large:
            a.copy_(b)


class Episodes:
    """A serving loop with its episodes; its staging thread ends with the object."""

    def __init__(self, case: dict, seed: int):
        self.server = Server(rows=65536)
        g = np.random.default_rng(case["episodes"])
        ticks = np.floor(np.exp(g.uniform(math.log(case["min_ticks"]), math.log(case["ticks"] + 1), case["episodes"])))
        self.episodes = []
        for e, (ships, k) in enumerate(zip(_ragged(case["episodes"], case["ships"]).tolist(), ticks.tolist())):
            world = flight_worlds(seed * 1_000_033 + e, 1, ships)
            world.packed()                       # the request in columns, as its client makes it
            self.episodes.append(Episode(e, world, int(k)))

    def __del__(self):
        self.server.close()


FLIGHT_OUT = ("pos", "vel", "goto", "last_g", "last_collision", "speed_fraction", "follow_range", "effect_stamp",
              "follow_id", "owner_id", "clock", "mode", "massive", "sensor")
TURN_OUT = ("rot", "ang_vel", "torque", "rot_roll")
COMBAT_OUT = ("formation_slots", "owner_ptr", "hits_n", "ev_n", "ev_self", "flags")
COMPOSED_OUT = ("last_c", "level", "key", "mod", "hits")
COLLIDE_STATE = ("pos", "vel", "old_pos", "old_vel", "goto", "last_g", "last_c", "last_collision", "speed_fraction",
                 "mode", "level", "key", "mod")
COLLIDE_OUT = COLLIDE_STATE + ("hits_n", "hits", "imp_n", "imp_slot", "imp_s", "imp_closing")


def _planes(park, names) -> list:
    return [getattr(park, "_" + k) for k in names]


def prepare(case: dict, seed: int) -> dict:
    kind, dev = case["kind"], "cuda"
    g = np.random.default_rng(seed)
    st = {"case": case}
    if kind == "flight":
        sizes = _ragged(case["worlds"], case["ships"]) if case["ragged"] else np.full(case["worlds"], case["ships"])
        w = _flight_worlds(g, sizes)
        park = VecModesPark(w.n, device=dev, dynamical_orientation=case["orientation"], use_new_orbit=case["new_orbit"])
        w.load(park)
        w.apply(park)
        if case["masked"]:                       # a quarter of the worlds wait for their next tick
            st["active"] = torch.from_numpy(np.repeat(g.random(len(sizes)) < 0.75, sizes)).to(dev)
        else:
            st["graph"] = ModesGraph(park)
        keep = _planes(park, [k[1:] for k in park.row_tensors() if k != "refiled"])
        st["out"] = _planes(park, FLIGHT_OUT + (TURN_OUT if case["orientation"] else ()))
    elif kind == "serve":
        st["serving"] = Episodes(case, seed)
        return st
    elif kind == "collide":
        make = collide_statics_worlds if case["statics"] else collide_worlds
        W, T = case["worlds"], min(case["worlds"], TEMPLATES)
        if case["statics"]:
            w = make(seed, T, case["ships"], case["fixed"], case["statics"], ticks=1)
            N = case["ships"] + case["fixed"]
        else:
            w = make(seed, T, case["ships"], case["free"], case["fixed"], ticks=1)
            N = case["ships"] + case["free"] + case["fixed"]
        some = VecCollidePark(T, N, device=dev, statics=case["statics"])
        some.load(w.worlds, w.collidables)
        park = VecCollidePark(W, N, device=dev, statics=case["statics"])
        if case["statics"]:
            park._empty_statics(some.B)
        at = torch.arange(W, device=dev) % T     # the world that each of the park's worlds starts as
        for k, t in vars(some).items():
            if isinstance(t, torch.Tensor) and t.dim() > 1 and t.shape[0] == T:
                getattr(park, k).copy_(t[at])
        ships = torch.zeros(W, N, dtype=torch.bool, device=dev)
        ships[:, :case["ships"]] = True
        aim = case["ships"] + g.integers(0, N - case["ships"], (W, N)) if N > case["ships"] else np.zeros((W, N), np.int64)
        aim = torch.from_numpy(aim).to(dev)      # every ship flies at another ball of its world's rest
        park.goto_point(ships, park.pos.gather(1, aim[..., None].expand(W, N, 3)))
        st["graph"] = CollideGraph(park)
        keep = [getattr(park, k) for k in COLLIDE_STATE]
        st["out"] = [getattr(park, k) for k in COLLIDE_OUT]
    elif kind in ("combat", "composed"):
        w = _combat_worlds(g, case)
        cls = VecComposedPark if kind == "composed" else VecCombatPark
        park = cls(len(w.rows), device=dev, use_new_orbit=True)
        park.load(w.rows)
        w.apply(park)
        st["graph"] = CombatGraph(park)
        names = [k[1:] for k in park.row_tensors() if k != "refiled"]
        keep = _planes(park, names)
        st["out"] = _planes(park, FLIGHT_OUT + TURN_OUT + COMBAT_OUT + (COMPOSED_OUT if kind == "composed" else ()))
    elif kind == "server":
        W, K = case["worlds"], case["ships"]
        w = _server_worlds(g, W, K)
        park = VecModesPark(W * K, device=dev)
        park.load_columns(w["cols"])
        srv = server.VecServer(server.ModesAdapter(park), list(range(K)) * W, kernel="cuda")
        srv.pre_tick()                           # the first tick (every ship's addition) eagerly
        srv.evolve()
        srv.post_tick()
        graph = server.ServerGraph(srv, ["GotoDirection", "SetSpeedFraction"] * K)
        d = torch.from_numpy(w["direction"]).to(dev).reshape(W, K, 3)
        s = torch.from_numpy(w["speed"]).to(dev).reshape(W, K, 1)
        for k in range(K):
            for x, f in ((graph.inputs[2 * k], d[:, k]), (graph.inputs[2 * k + 1], s[:, k])):
                x["mask"].fill_(True)
                x["ball"].fill_(k + 1)
                x["f"][:, :f.shape[1]].copy_(f)
        st["graph"] = graph
        b = graph.out
        out = [b.stamp, b.clock, b.route, b.has_character, b.gets_bubble]
        keep = (_planes(park, [k[1:] for k in park.row_tensors() if k != "refiled"])
                + [park.cloaked, park.bubble, srv.stamp_for_system, srv._bubble_time, srv.dead, srv.settled, srv._fresh,
                   srv._listed])
        st["out"] = _planes(park, FLIGHT_OUT) + out
    else:                                        # the partition layer: every class a warp a world, small worlds a thread
        pw = _partition_worlds(case, seed)
        plan = {4: (1, 64)} if kind == "face" else {c: (32, 128) for c in (4, 8, 16, 32, 64, 128)}
        r = partition_setup(pw, torch.device(dev, torch.cuda.current_device()), ragged=True, plan=plan)
        park, part, srv = r["park"], r["part"], r["server"]
        st.update(graph=r["graph"], part=part, setup=r)
        keep = (_planes(park, [k[1:] for k in park.row_tensors() if k != "refiled"])
                + [park.cloaked, park.bubble, srv.stamp_for_system, srv._bubble_time, srv.dead, srv.settled, srv._fresh,
                   srv._listed] + [t for layer, _ in part.layers for t in layer.st.values()])
        st["out"] = _planes(park, FLIGHT_OUT) + [layer.st[k] for layer, _ in part.layers
                                                 for k in ("level", "key", "bubble", "slen")]
        st["ev"] = [(layer.st["ev"], layer.st["evn"], torch.arange(layer.M, device=park.dev)[:, None])
                    for layer, _ in part.layers]
    st["park"] = park
    st["start"] = Snapshot(keep)
    return st


def _serve(s: Episodes) -> list:
    """Every episode submitted at once, run to its end; each one's final state, in the order of the episodes."""
    srv = s.server
    srv.results.clear()
    srv.reset_stats()
    serve(srv, s.episodes, realtime=False)
    done = [srv.results[e.eid] for e in s.episodes]
    return [torch.cat([r.field(k) for r in done]) for k in ("pos", "vel", "goto", "rot", "ang_vel", "clock", "mode",
                                                            "follow_id", "effect_stamp")]


def run(state: dict) -> list:
    case = state["case"]
    if case["kind"] == "serve":
        return _serve(state["serving"])
    state["start"].restore()
    if "active" in state:
        for _ in range(case["ticks"]):
            state["park"].evolve(active=state["active"])
    else:
        tick = state["graph"].tick
        for _ in range(case["ticks"]):
            tick()
    out = list(state["out"])
    if "ev" in state:                            # the last tick's events, world by world, in their order
        out += [torch.where(at < n, ev, 0) for ev, n, at in state["ev"]]
        out.append(state["part"].event_counts())
    return out


# ============================================================================ what a pass cannot do without

def work(case: dict) -> dict:
    """Bytes: the state that a tick reads and writes, each field once a tick (the ticks are calls of their own: the
    state lives in memory between them). Operations: the arithmetic of the ships' laws a tick, by kind."""
    kind, ticks = case["kind"], case["ticks"]
    mean = lambda most: (most - 1) / math.log(most) if most > 1 else 1.0      # of a log-uniform size
    if kind == "flight":
        n = case["worlds"] * (mean(case["ships"]) if case["ragged"] else case["ships"]) * (0.75 if case["masked"] else 1)
        b, f = (503, 3000) if case["orientation"] else (346, 300)
    elif kind == "serve":
        n, b, f = case["episodes"] * mean(case["ships"]), 503, 3000
        ticks = (case["ticks"] - case["min_ticks"]) / math.log(case["ticks"] / case["min_ticks"])
    elif kind == "collide":
        n = case["worlds"] * (case["ships"] + case["free"] + case["fixed"])
        b, f = 560 + 75 * case["statics"], 600 + 400 * case["statics"]
    elif kind in ("combat", "composed"):
        n = case["worlds"] * (case["ships"] + case["missiles"] + case["spheres"])
        b, f = (553, 3000) if kind == "combat" else (665, 3500)
    elif kind == "server":
        n, b, f = case["worlds"] * case["ships"], 372 + 346, 350
    else:
        n = case["worlds"] * (mean(case["ships"]) if kind == "partition" else case["ships"])
        b, f = 476 + 372 + 346, 943 + 350
    return {"bytes": float(n * b * ticks), "flops": float(n * f * ticks)}


# ============================================================================ the pilots' flights in 64 bits

def exact(case: dict, seed: int):
    """The piloted cases' positions, velocities, goto points and thrusts: a ship at rest, its first tick at rest, then
    each tick the goto point 1e17 m along its pilot's direction from where it is, the full thrust toward it and the closed
    form of m v' = m a - k v over one second."""
    if case["kind"] == "server":
        w = _server_worlds(np.random.default_rng(seed), case["worlds"], case["ships"])
        cols, direction, speed = w["cols"], w["direction"], w["speed"]
    elif case["kind"] in ("partition", "face"):
        w = _partition_worlds(case, seed)
        cols, direction, speed = w.cols, w.direction, w.speed
    else:
        return None
    member = lambda x: x.astype(np.float32).astype(np.float64)       # the members that hold floats
    k, m = 1e6, cols["mass"] * member(cols["agility"])
    unit = direction / np.linalg.norm(direction, axis=1, keepdims=True)
    a = unit * (k * member(speed) * member(cols["max_vel"]) / m)[:, None]
    fall = np.exp(-k / m)[:, None]
    p, v, m = cols["pos"].copy(), np.zeros_like(cols["pos"]), m[:, None]
    for _ in range(case["ticks"]):
        goal = p + unit * 1e17
        p = p + m / k * (a - (v - m * a / k) * (fall - 1.0))
        v = m * a / k + (v - m * a / k) * fall
    layers = 0
    if case["kind"] != "server":
        sizes = w.sizes
        layers = len({next(c for c in (4, 8, 16, 32, 64, 128) if s <= c) for s in set(sizes.tolist())})
    rest = [None] * (len(FLIGHT_OUT) - 4 + (5 if case["kind"] == "server" else 5 * layers + 1))
    return [np.ascontiguousarray(x.T) for x in (p, v, goal, a)] + rest
