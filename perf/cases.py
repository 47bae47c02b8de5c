"""Performance cases: what a program that uses this framework has it do.

Every case goes through the public Python API (htrip_b200.minplus_oracle) on
seeded maps of the kinds the repository's workloads use (street-like grids and
mazes, htrip_b200/workloads.py).  The kinds of pass:

distance   one queryDistance call: a reachability / cost check between two cells
query      one queryAllPairs call, host viewpoints and host result
query_dev  one queryAllPairsDevice call, viewpoints and result in GPU memory
explore    one exploration step: the cells a robot team has just seen are
           opened (onBatchCellsOpened), then the distances between robots and
           frontier cells are asked for (a full query, or an incremental one
           over fixed watch points)
obstacle   a moving obstacle takes one step: the cells it leaves are opened, the
           leaves under its new footprint are rebuilt (onBatchLeavesChanged),
           then a query
weights    the traversal weights of one tile change (onTileWeightsChanged), then
           a query
build      a map is indexed from scratch (build), then its first query
fleet      many maps served together: one Batch.open and one Batch.query

``listed()`` names one case for each place of the range that a user meets;
``draw`` gives further ones of the same ranges.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from htrip_b200 import workloads as W
from htrip_b200.minplus_oracle import Batch, GridMap, HierarchyConfig, IncrementalState, MinPlusOracle

INF = 60000
ROBOTS = 4  # robots of an exploring team
SENSOR = 24  # sensor radius (cells) of the first observation, smaller on small maps


def _case(kind, rows, cols, b, k, *, g=2, corridor=0, m=0, steps=0, incremental=False, maps=0, name=None):
    """One case.  corridor 0: a street-like map, else a maze of that corridor
    width; k viewpoints; m cells opened per step (explore, fleet), footprint
    radius (obstacle); steps of the prepared mission; maps of a fleet."""
    c = dict(kind=kind, rows=rows, cols=cols, b=b, g=g, corridor=corridor, k=k, m=m, steps=steps,
             incremental=incremental, maps=maps)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: is one cell reachable from another, and how far
        _case("distance", 256, 256, 16, 2, name="distance_street256"),
        # a small robot team on an ordinary street map
        _case("query", 256, 256, 16, 16, name="query_street256_k16"),
        # the headline query: many goals in a narrow maze, long distances
        _case("query", 512, 512, 16, 256, corridor=1, name="query_maze512_k256"),
        # a planner that keeps its viewpoints and the matrix on the GPU; wide corridors
        _case("query_dev", 512, 512, 16, 64, corridor=16, name="query_dev_maze512_k64"),
        # the largest query: hundreds of goals on a big map whose sides are no multiple of the tile
        _case("query_dev", 1000, 1013, 16, 509, name="query_dev_street1000_k509"),
        # exploration of a large map in large steps, each followed by a query
        _case("explore", 1024, 1024, 8, 64, m=256, steps=1000, name="explore_street1024_m256"),
        # exploration of a small odd-sized map in small steps, fixed watch points
        _case("explore", 300, 277, 8, 33, m=24, steps=1000, incremental=True, name="explore_street300_m24_incr"),
        # a vehicle drives through a mapped area
        _case("obstacle", 512, 512, 16, 32, m=3, steps=24, name="obstacle_street512"),
        # terrain costs of one tile are revised
        _case("weights", 256, 256, 8, 32, steps=24, name="weights_street256"),
        # a small map is loaded
        _case("build", 250, 256, 16, 16, name="build_street250"),
        # a large map is loaded
        _case("build", 1024, 1024, 8, 128, name="build_street1024"),
        # many maps of mixed sizes and tile sides updated and queried together
        _case("fleet", 0, 0, 0, 128, m=64, steps=300, maps=16, name="fleet16"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(("distance", "query", "query", "query_dev", "query_dev", "explore", "explore", "explore",
                       "obstacle", "weights", "build", "build", "fleet"))
    if kind == "fleet":
        return _case("fleet", 0, 0, 0, _log(rng, 16, 128), m=_log(rng, 8, 64), steps=300, maps=rng.randint(3, 16))
    most = 640 if kind in ("weights", "obstacle") else 1024
    rows, cols = _log(rng, 80, most), 0
    cols = max(64, min(most, int(rows * rng.uniform(0.75, 1.0))))
    g = 4 if max(rows, cols) <= 128 and rng.random() < 0.5 else 2
    b = rng.choice((4, 8)) if g == 4 else rng.choice((8, 8, 16, 16, 32))
    corridor = rng.choice((0, 0, 1, rng.randint(2, 16)))
    if kind == "distance":
        return _case(kind, rows, cols, b, 2, g=g, corridor=corridor)
    if kind in ("query", "query_dev"):
        return _case(kind, rows, cols, b, _log(rng, 3, 512), g=g, corridor=corridor)
    if kind == "explore":
        return _case(kind, rows, cols, b, _log(rng, 6, 128), g=g, m=_log(rng, 1, 384), steps=500,
                     incremental=rng.random() < 0.4)
    if kind == "obstacle":
        return _case(kind, rows, cols, b, _log(rng, 4, 64), g=g, m=rng.randint(1, 6), steps=24)
    if kind == "weights":
        return _case(kind, rows, cols, min(b, 16), _log(rng, 4, 64), g=g, steps=24)
    return _case(kind, rows, cols, b, _log(rng, 4, 128), g=g, corridor=corridor)


# ---------------------------------------------------------------------------
# Inputs (host data made from the case and the seed alone).
# ---------------------------------------------------------------------------
def _truth(case, seed):
    side = max(case["rows"], case["cols"])
    if case["corridor"]:
        grid = W.maze_grid(side, case["corridor"], seed)
    else:
        grid = W.street_grid(side, seed, rect_min=4, rect_max=max(8, min(40, side // 8)))
    return np.ascontiguousarray(grid[:case["rows"], :case["cols"]])


def _mission(case, seed):
    """A team explores a map: the first observation, the cells opened at each
    step and the viewpoints asked for after it."""
    truth = _truth(case, seed)
    m, k, steps = case["m"], case["k"], case["steps"]
    radius = min(SENSOR, max(truth.shape) // 10)
    observed0, starts, batches = W.exploration_stream(truth, ROBOTS, radius, m, steps, seed + 1)
    if len(batches) > 1 and len(batches[-1]) < m:
        batches.pop()  # the last few cells
    if case["incremental"]:  # fixed watch points in the first observation
        vps = [W.sample_free(observed0, k, seed + 2)] * len(batches)
    else:  # the robots and cells of the current frontier
        order = np.concatenate([starts] + batches)
        vps = []
        for i in range(len(batches)):
            end = len(starts) + (i + 1) * m
            recent = order[max(0, end - 4 * k):end]
            pick = np.linspace(0, len(recent) - 1, max(1, min(len(recent), k - len(starts)))).astype(np.int64)
            vps.append(np.ascontiguousarray(np.concatenate([starts, recent[pick]])[:k]))
    return dict(observed0=observed0, batches=batches, vps=vps)


def _fleet_cases(case):
    """The fleet's maps: mixed sides, tile sides, step sizes and viewpoint
    counts, the same for every seed (the maps themselves differ)."""
    r = random.Random(case["maps"] * 1000003 + case["k"] * 1009 + case["m"])
    out = []
    for i in range(case["maps"]):
        side = _log(r, 64, 320)
        out.append(_case("explore", side, max(64, side - r.randint(0, 40)), r.choice((8, 16, 16)),
                         _log(r, 8, case["k"]), m=_log(r, 4, case["m"]), steps=case["steps"]))
    return out


def _inputs(case, seed):
    kind = case["kind"]
    if kind == "fleet":
        return [_mission(c, seed * 100 + i) for i, c in enumerate(_fleet_cases(case))]
    if kind == "explore":
        return _mission(case, seed)
    truth = _truth(case, seed)
    rng = np.random.default_rng(seed + 3)
    inp = dict(grid=truth, vps=W.sample_free(truth, case["k"], seed + 2))
    if kind == "obstacle":
        rad = case["m"]
        yy, xx = np.mgrid[-rad:rad + 1, -rad:rad + 1]
        disc = np.stack([yy, xx], axis=-1)[yy * yy + xx * xx <= rad * rad]
        foot, leaves = [], []
        lx = _leaves_x(case)
        for p in W.sample_free(truth, case["steps"], seed + 4):
            cells = p + disc
            cells = cells[(cells >= 0).all(1) & (cells[:, 0] < truth.shape[0]) & (cells[:, 1] < truth.shape[1])]
            cells = np.ascontiguousarray(cells[truth[cells[:, 0], cells[:, 1]] == W.FREE]).astype(np.int32)
            foot.append(cells)
            leaves.append(np.unique(cells[:, 0] // case["b"] * lx + cells[:, 1] // case["b"]).astype(np.int32))
        inp.update(foot=foot, leaves=leaves)
    if kind == "weights":
        b = case["b"]
        inp["weights"] = rng.integers(1, 10, size=truth.shape).astype(np.uint16)
        changes = []
        for r, c in W.sample_free(truth, case["steps"], seed + 4):
            ty, tx = int(r) // b, int(c) // b
            free = [(y, x) for y in range(ty * b, min(truth.shape[0], (ty + 1) * b))
                    for x in range(tx * b, min(truth.shape[1], (tx + 1) * b)) if truth[y, x] == W.FREE]
            changes.append((tx, ty, [(p, int(w)) for p, w in zip(free, rng.integers(1, 10, size=len(free)))]))
        inp["changes"] = changes
    return inp


def _leaves_x(case):
    S = case["b"]
    while S < max(case["rows"], case["cols"]):
        S *= case["g"]
    return S // case["b"]


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def _oracle(case, grid):
    o = MinPlusOracle(HierarchyConfig(case["b"], case["g"], case["g"]))
    if not o.build(grid):
        raise RuntimeError("build refused the map")
    return o


class _Explorer:
    """A robot team's map: its index, what it has seen so far, its next steps."""

    def __init__(self, case, mission):
        self.mission = mission
        self.grid = GridMap(mission["observed0"].copy())
        self.oracle = _oracle(case, self.grid)
        self.incremental = IncrementalState() if case["incremental"] else None
        self.step = 0

    def next(self):
        """The cells the next step opens (already marked Free) and its viewpoints."""
        if self.step == len(self.mission["batches"]):  # everything seen: a new mission on the same map
            self.grid.observed[...] = self.mission["observed0"]
            self.oracle.build(self.grid)
            self.step = 0
        cells, vps = self.mission["batches"][self.step], self.mission["vps"][self.step]
        self.grid.observed[cells[:, 0], cells[:, 1]] = W.FREE
        self.step += 1
        return cells, vps

    def stats(self):
        st = self.oracle.last_batch_stats
        return [st.n_touched_leaves, st.n_dirty_ancestors, st.n_pivots]


def prepare(case, seed):
    kind = case["kind"]
    inp = _inputs(case, seed)
    state = dict(kind=kind, step=0)
    if kind == "fleet":
        state["batch"] = Batch()
        state["teams"] = [_Explorer(c, i) for c, i in zip(_fleet_cases(case), inp)]
        return state
    if kind == "explore":
        state["team"] = _Explorer(case, inp)
        return state
    state.update(inp)
    if kind == "build":
        state["grid"] = GridMap(inp["grid"])
        state["oracle"] = MinPlusOracle(HierarchyConfig(case["b"], case["g"], case["g"]))
        return state
    state["grid"] = GridMap(inp["grid"], inp.get("weights"))
    if kind == "weights":
        state["grid"].weights = inp["weights"].copy()
    if kind == "obstacle":
        f = inp["foot"][0]
        state["grid"].observed = inp["grid"].copy()
        state["grid"].observed[f[:, 0], f[:, 1]] = W.OBSTACLE
    state["oracle"] = _oracle(case, state["grid"])
    if kind == "query_dev":
        vps = inp["vps"]
        state["vps_dev"] = torch.from_numpy(vps).cuda()
        state["pass_dev"] = torch.ones(len(vps), dtype=torch.uint8, device="cuda")
        state["out_dev"] = torch.empty((len(vps), len(vps)), dtype=torch.uint16, device="cuda")
        torch.cuda.synchronize()
    return state


def run(state):
    kind = state["kind"]
    if kind == "distance":
        a, c = state["vps"]
        return state["oracle"].queryDistance(a, c, state["grid"])
    if kind == "query":
        return state["oracle"].queryAllPairs(state["vps"], state["grid"])
    if kind == "query_dev":
        state["oracle"].queryAllPairsDevice(state["vps_dev"].data_ptr(), state["pass_dev"].data_ptr(),
                                            len(state["vps_dev"]), state["out_dev"].data_ptr())
        return state["out_dev"]
    if kind == "build":
        state["oracle"].build(state["grid"])
        return state["oracle"].queryAllPairs(state["vps"], state["grid"])
    if kind == "explore":
        t = state["team"]
        cells, vps = t.next()
        t.oracle.onBatchCellsOpened(cells, t.grid)
        if t.incremental is not None:
            d = t.oracle.queryAllPairsIncremental(vps, t.grid, t.incremental)
        else:
            d = t.oracle.queryAllPairs(vps, t.grid)
        return {"distances": d, "stats": t.stats()}
    if kind == "fleet":
        nxt = [t.next() for t in state["teams"]]
        state["batch"].open([(t.oracle, cells, t.grid) for t, (cells, _) in zip(state["teams"], nxt)])
        d = state["batch"].query([(t.oracle, vps, t.grid) for t, (_, vps) in zip(state["teams"], nxt)])
        return {"distances": d, "stats": np.array([t.stats() for t in state["teams"]])}
    o, grid, i = state["oracle"], state["grid"], state["step"]
    if kind == "obstacle":
        old = state["foot"][i]
        i = (i + 1) % len(state["foot"])
        new = state["foot"][i]
        grid.observed[old[:, 0], old[:, 1]] = W.FREE
        o.onBatchCellsOpened(old, grid)
        grid.observed[new[:, 0], new[:, 1]] = W.OBSTACLE
        o.onBatchLeavesChanged(state["leaves"][i], grid)
    else:  # weights
        tx, ty, cells = state["changes"][i]
        i = (i + 1) % len(state["changes"])
        o.onTileWeightsChanged(tx, ty, cells, grid)
    state["step"] = i
    return o.queryAllPairs(state["vps"], grid)


# ---------------------------------------------------------------------------
# exact: breadth-first search / relaxation on the grid itself
# ---------------------------------------------------------------------------
def _bfs(grid, vps, limit_s=12.0):
    """(k, k) int64 unit-cost distances between cells of a grid, in chunks of
    sources; None when it would take long."""
    import time

    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t0 = time.perf_counter()
    free = torch.from_numpy(grid == W.FREE).to(dev)
    v = torch.from_numpy(np.asarray(vps)).long().to(dev)
    k, (R, C) = len(v), free.shape
    out = torch.full((k, k), INF, dtype=torch.int64, device=dev)
    for s0 in range(0, k, 64):
        s = v[s0:s0 + 64]
        n = len(s)
        front = torch.zeros((n, R, C), dtype=torch.bool, device=dev)
        front[torch.arange(n, device=dev), s[:, 0], s[:, 1]] = True
        front &= free
        seen = front.clone()
        d = 0
        while d < INF:
            hit = front[:, v[:, 0], v[:, 1]]
            out[s0:s0 + n][hit] = d
            nxt = torch.zeros_like(front)
            nxt[:, 1:] |= front[:, :-1]
            nxt[:, :-1] |= front[:, 1:]
            nxt[:, :, 1:] |= front[:, :, :-1]
            nxt[:, :, :-1] |= front[:, :, 1:]
            nxt &= free & ~seen
            seen |= nxt
            front = nxt
            d += 1
            if d % 32 == 0:
                if not bool(front.any()):
                    break
                if time.perf_counter() - t0 > limit_s:
                    return None
    return out.cpu()


def _relax(grid, weights, vps, limit_s=12.0):
    """(k, k) int64 weighted distances: an edge costs max(1, (w_u + w_v) // 2)."""
    import time

    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t0 = time.perf_counter()
    free = torch.from_numpy(grid == W.FREE).to(dev)
    w = torch.from_numpy(weights.astype(np.int64)).to(dev)
    far = 1 << 40

    def edge(a, c, fa, fc):
        return torch.where(fa & fc, torch.clamp((a + c) // 2, min=1), far)

    down, right = edge(w[1:], w[:-1], free[1:], free[:-1]), edge(w[:, 1:], w[:, :-1], free[:, 1:], free[:, :-1])
    v = torch.from_numpy(np.asarray(vps)).long().to(dev)
    k = len(v)
    d = torch.full((k,) + tuple(free.shape), far, dtype=torch.int64, device=dev)
    d[torch.arange(k, device=dev), v[:, 0], v[:, 1]] = 0
    for it in range(1 << 20):
        old = d.clone() if it % 32 == 0 else None
        d[:, 1:] = torch.minimum(d[:, 1:], d[:, :-1] + down)
        d[:, :-1] = torch.minimum(d[:, :-1], d[:, 1:] + down)
        d[:, :, 1:] = torch.minimum(d[:, :, 1:], d[:, :, :-1] + right)
        d[:, :, :-1] = torch.minimum(d[:, :, :-1], d[:, :, 1:] + right)
        if old is not None and torch.equal(old, d):
            break
        if it % 32 == 0 and time.perf_counter() - t0 > limit_s:
            return None
    return torch.clamp(d[:, v[:, 0], v[:, 1]], max=INF).cpu()


def exact(case, seed):
    kind = case["kind"]
    if case["corridor"] and case["corridor"] < 3:  # paths of tens of thousands of steps: minutes
        return None
    inp = _inputs(case, seed)
    if kind in ("explore", "fleet"):
        got = []
        for m in inp if kind == "fleet" else [inp]:
            obs = m["observed0"].copy()
            cells = m["batches"][0]
            obs[cells[:, 0], cells[:, 1]] = W.FREE
            d = _bfs(obs, m["vps"][0], 4.0 if kind == "fleet" else 12.0)
            if d is None:
                return None
            got.append(d)
        return {"distances": got if kind == "fleet" else got[0], "stats": None}
    grid, vps = inp["grid"], inp["vps"]
    if kind == "obstacle":
        grid = grid.copy()
        f = inp["foot"][1 % len(inp["foot"])]
        grid[f[:, 0], f[:, 1]] = W.OBSTACLE
    if kind == "weights":
        for p, w in inp["changes"][0][2]:
            inp["weights"][p] = w
        return _relax(grid, inp["weights"], vps)
    d = _bfs(grid, vps)
    if d is None:
        return None
    return int(d[0, 1]) if kind == "distance" else d


# ---------------------------------------------------------------------------
# work: what a pass cannot do without
# ---------------------------------------------------------------------------
def _levels(case):
    """Per internal level: (nodes, matrix order, ports per child)."""
    b, g = case["b"], case["g"]
    S = _leaves_x(case) * b
    out, cs = [], b
    while cs < S:
        side = cs * g
        out.append(((S // side) ** 2, g * g * (4 * cs - 4), 4 * cs - 4))
        cs = side
    return out


def _query_work(case, k):
    """Viewpoint rows of the leaves, then per level the matrix rows under the
    children that hold a viewpoint, each viewpoint combined with them once
    (an addition and a minimum per entry); the result written."""
    nbytes, flops = k * (4 * case["b"] - 4) * 2 + 2 * k * k, 0
    for nodes, n, ports in _levels(case):
        children = nodes * case["g"] ** 2
        held = children * (1 - (1 - 1 / children) ** k)
        nbytes += 2 * held * ports * n / 2
        flops += 2 * k * ports * n / 2
    return nbytes, flops


def _open_work(case, m):
    """Per level the matrices above the opened cells (up to the robots' number)
    closed over as many pivots as cells: half of each symmetric matrix."""
    dirty = min(ROBOTS, max(1, m))
    b2 = case["b"] ** 2
    nbytes = dirty * b2 * b2 * 2
    flops = 2 * dirty * b2 * b2 / 2 * min(m, b2)
    for nodes, n, _ in _levels(case):
        d = min(nodes, dirty)
        nbytes += d * n * n * 2
        flops += 2 * d * n * n / 2 * min(m, n / 4)
    return nbytes, flops


def _node_work(n):
    """One internal matrix from its children and seams, once the pivots (about
    a quarter of its order lies on seams): the pivots' own closure, then each
    half of the symmetric matrix through the pivots of one child."""
    return 2 * n * n, 2 * n ** 3 * (1 / 64 + 1 / 64 + 1 / 32)


def work(case):
    kind, k = case["kind"], case["k"]
    if kind == "fleet":
        got = [work(c) for c in _fleet_cases(case)]
        return {key: sum(w[key] for w in got) for key in ("bytes", "flops")}
    nbytes, flops = _query_work(case, k)
    more = []
    if kind == "explore":
        more.append(_open_work(case, case["m"]))
    if kind in ("obstacle", "weights"):  # one leaf and every matrix above it
        more += [_node_work(n) for _, n, _ in _levels(case)] + [(case["b"] ** 4 * 2, 0)]
        if kind == "obstacle":
            more.append(_open_work(case, case["m"] ** 2 * 3))
    if kind == "build":
        more.append((_leaves_x(case) ** 2 * case["b"] ** 4 * 2, 0))
        for nodes, n, _ in _levels(case):
            nb, fl = _node_work(n)
            more.append((nodes * nb, nodes * fl))
    return {"bytes": float(nbytes + sum(b for b, _ in more)), "flops": float(flops + sum(f for _, f in more))}
