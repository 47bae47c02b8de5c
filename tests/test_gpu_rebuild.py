"""A handle that is built again, and rebuilds in place: what earlier calls left
behind (flags of a failed opening, a trace, scratch memory, weights, an
incremental state) reaches no later result.  Matrices, statistics and distances
against the CPU restatement of the reference, tolerance 0."""
import threading

import numpy as np
import pytest

from helpers import FREE, OBST, make_grid
from htrip_b200 import workloads as W
from oracle.ref import PortOracle, port_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not port_available(), reason="oracle port not built (make -C oracle port)")]


def _stats(dev):
    st = dev.last_batch_stats
    return st.n_touched_leaves, st.n_dirty_ancestors, st.n_pivots


@pytest.mark.parametrize("kind,side,b,g", [("noise", 64, 16, 2), ("street", 100, 8, 2), ("noise", 54, 9, 3)])
def test_build_on_a_handle_clears_flags_of_a_failed_opening(gpu, kind, side, b, g):
    from htrip_b200.minplus_oracle import HierarchyConfig, MinPlusOracle, selftest_stale_flags
    observed, cells = W.withheld_open(make_grid(kind, side, side, b), 30, 5)
    dev, new, cpu = MinPlusOracle(HierarchyConfig(b, g, g)), MinPlusOracle(HierarchyConfig(b, g, g)), PortOracle(b, g)
    assert dev.build(observed) and new.build(observed) and cpu.build(observed)
    selftest_stale_flags(dev)
    assert dev.build(observed)
    observed[cells[:, 0], cells[:, 1]] = FREE
    for o in (dev, new):
        o.onBatchCellsOpened(cells, observed)
    cpu.open_batch(cells, observed)
    assert _stats(dev) == cpu.stats()
    assert dev.lastOpenLevels() == new.lastOpenLevels()
    assert dev.stateDigest() == new.stateDigest()


@pytest.mark.parametrize("change", ["build", "blocked", "leaves", "weight"])
def test_no_opening_trace_after_a_rebuild(gpu, change):
    """The trace's device memory is the rebuild's staging: it is not read afterwards."""
    from htrip_b200.minplus_oracle import HierarchyConfig, HtripError, MinPlusOracle
    observed, cells = W.withheld_open(make_grid("noise", 64, 64, 3), 20, 5)
    dev = MinPlusOracle(HierarchyConfig(16, 2, 2))
    assert dev.build(observed)
    observed[cells[:, 0], cells[:, 1]] = FREE
    dev.onBatchCellsOpened(cells, observed)
    assert len(dev.lastOpenTrace()) > 0
    p = tuple(int(x) for x in cells[0])
    if change == "build":
        assert dev.build(observed)
    elif change == "blocked":
        observed[p] = OBST
        dev.onCellBlocked(p, observed)
    elif change == "leaves":
        dev.onBatchLeavesChanged([0], observed)
    else:
        dev.onCellWeightChanged(p, 5, observed)
    with pytest.raises(HtripError, match="no device-driven opening"):
        dev.lastOpenTrace()


def test_indexes_of_several_tile_sides_build_at_once(gpu):
    """Threads with an index each: one's launches do not set limits for the other's."""
    from htrip_b200.minplus_oracle import HierarchyConfig, MinPlusOracle
    errors, digests = [], {}

    def work(b):
        try:
            grid = make_grid("noise", 2 * b, 2 * b, b)
            dev = MinPlusOracle(HierarchyConfig(b, 2, 2))
            assert dev.build(grid)
            digests[b] = dev.stateDigest()
            for _ in range(2000):
                assert dev.build(grid)
            assert dev.stateDigest() == digests[b]
        except Exception as e:  # noqa: BLE001 (reported below)
            errors.append((b, repr(e)))

    threads = [threading.Thread(target=work, args=(b,)) for b in (10, 16, 11, 15)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert errors == []


@pytest.mark.parametrize("side,b,g", [(512, 8, 2), (500, 32, 2), (486, 6, 3)])
def test_build_scratch_is_given_back(gpu, side, b, g):
    """An index holds its estimate, the staged grid and small tables: per node at most
    64 bytes of state, per level a few blocks of 256 bytes, lists of a call's leaves and nodes."""
    from htrip_b200.minplus_oracle import HierarchyConfig, MinPlusOracle, estimate_bytes
    cfg = HierarchyConfig(b, g, g)
    grid = make_grid("noise", side, side, 1)
    dev = MinPlusOracle(cfg)
    assert dev.build(grid)
    nodes = dev.num_leaf_tiles_x ** 2 * g * g // (g * g - 1) + 1
    bound = estimate_bytes(cfg, side, side) + dev.S ** 2 + 64 * nodes + (dev.H + 1) * 16 * 256 + 65536
    assert dev.deviceMemoryBytes() <= bound
    p = tuple(int(x) for x in np.argwhere(grid == FREE)[100])
    grid[p] = OBST
    dev.onCellBlocked(p, grid)
    assert dev.deviceMemoryBytes() <= bound


def _same_matrices(dev, cpu):
    for i in range(dev.num_leaf_tiles_x ** 2):
        assert np.array_equal(dev.leaf_D(i), cpu.leaf_D(i)), f"leaf {i}"
    for lvl in range(1, dev.H + 1):
        for n in range(dev.level_dims(lvl)[3]):
            assert np.array_equal(dev.node_DU(lvl, n), cpu.node_DU(lvl, n)), f"level {lvl} node {n}"


def _weighted_distances(grid, wts, vps):
    """Dijkstra over the passable cells, an edge costing max(1, (w_u + w_v) / 2)."""
    from scipy.sparse import coo_matrix
    from scipy.sparse.csgraph import dijkstra

    from htrip_b200.minplus_oracle import INF
    idx = np.arange(grid.size).reshape(grid.shape)
    ends, cost = [], []
    for a, c in ((np.s_[1:], np.s_[:-1]), (np.s_[:, 1:], np.s_[:, :-1])):
        ok = (grid[a] == FREE) & (grid[c] == FREE)
        ends.append(np.stack([idx[a][ok], idx[c][ok]]))
        cost.append(np.maximum(1, (wts[a][ok].astype(int) + wts[c][ok]) // 2))
    ends, cost = np.concatenate(ends, axis=1), np.concatenate(cost)
    graph = coo_matrix((cost, (ends[0], ends[1])), shape=(grid.size, grid.size)).tocsr()
    at = idx[vps[:, 0], vps[:, 1]]
    return np.minimum(dijkstra(graph, directed=False, indices=at)[:, at], INF).astype(np.uint16)


@pytest.mark.parametrize("b,g,sizes", [
    (8, 2, ((64, 64), (40, 61), (33, 64))),      # one padded side
    (16, 2, ((120, 128), (65, 20), (128, 128))),
    (5, 3, ((45, 45), (16, 40), (30, 44))),
    (8, 2, ((64, 64), (70, 64), (10, 12), (64, 33))),   # padded sides 64, 128, 16, 64
])
def test_one_handle_built_again_and_again(gpu, b, g, sizes):
    """Per map: every matrix, an opening with its statistics, queries (an incremental
    state that outlives the map among them), a blocked cell; then with weights and
    without them again; then after root growth and after an offload."""
    from htrip_b200.minplus_oracle import HierarchyConfig, IncrementalState, MinPlusOracle
    dev, state = MinPlusOracle(HierarchyConfig(b, g, g)), IncrementalState()
    for turn, (rows, cols) in enumerate(sizes):
        truth = make_grid("noise", rows, cols, rows + turn)
        observed, cells = W.withheld_open(truth, 40, turn)
        cpu = PortOracle(b, g)
        assert dev.build(observed) and cpu.build(observed)
        _same_matrices(dev, cpu)
        vps = W.sample_free(observed, 9, turn)
        assert np.array_equal(dev.queryAllPairsIncremental(vps, observed, state), cpu.query(vps, observed))
        for part in (cells[:15], cells[15:]):
            observed[part[:, 0], part[:, 1]] = FREE
            dev.onBatchCellsOpened(part, observed)
            cpu.open_batch(part, observed)
            assert _stats(dev) == cpu.stats()
            assert np.array_equal(dev.queryAllPairsIncremental(vps, observed, state), cpu.query(vps, observed))
        _same_matrices(dev, cpu)
        wts = np.random.default_rng(turn).integers(1, 30, size=observed.shape).astype(np.uint16)
        assert dev.build(observed, weights=wts)
        assert np.array_equal(dev.queryAllPairs(vps, observed), _weighted_distances(observed, wts, vps))
        p = tuple(int(x) for x in vps[0])
        observed[p] = OBST
        cpu = PortOracle(b, g)
        assert dev.build(observed) and cpu.build(observed)
        _same_matrices(dev, cpu)
    big = np.full((dev.S * g, dev.S * g), OBST, np.uint8)
    big[:observed.shape[0], :observed.shape[1]] = observed
    dev.liftRoot(big)
    assert dev.build(big) and cpu.build(big)
    _same_matrices(dev, cpu)
    dev.offload()
    assert dev.build(observed) and cpu.build(observed)
    _same_matrices(dev, cpu)


@pytest.mark.parametrize("side,b,g", [(64, 4, 2), (96, 8, 2), (100, 9, 2), (128, 16, 2), (128, 32, 2), (54, 6, 3)])
def test_leaves_and_weights_changed(gpu, side, b, g):
    """onBatchLeavesChanged (the parents to rebuild are chosen on the device),
    onCellWeightChanged and onTileWeightsChanged against a build of the changed map (the
    two agree here; in general an unchanged exterior hides a changed seam higher up, as in
    the reference)."""
    from htrip_b200.minplus_oracle import GridMap, HierarchyConfig, MinPlusOracle
    rng = np.random.default_rng(side + b)
    grid = make_grid("street", side, side, b)
    dev, cpu = MinPlusOracle(HierarchyConfig(b, g, g)), PortOracle(b, g)
    assert dev.build(grid)
    lx = dev.num_leaf_tiles_x
    for n in (1, 4, 12):
        at = rng.choice(side * side, size=n, replace=False)
        r, c = at // side, at % side
        grid[r, c] = np.where(grid[r, c] == FREE, OBST, FREE)
        leaves = np.unique(r // b * lx + c // b)
        dev.onBatchLeavesChanged(np.concatenate([leaves, [0]]), grid)  # leaf 0 may be unchanged
        assert cpu.build(grid)
        _same_matrices(dev, cpu)
    vps = W.sample_free(grid, 24, 3)
    gm, new = GridMap(grid, np.ones(grid.shape, np.uint16)), MinPlusOracle(HierarchyConfig(b, g, g))
    assert dev.build(gm)
    for turn, w in enumerate((7, 400, 60000, 1)):
        p = tuple(int(x) for x in vps[turn % 2])
        dev.onCellWeightChanged(p, w, gm)
        ty, tx = (int(x) // b for x in vps[2 + turn])
        box = [(r, c) for r in range(ty * b, min(side, ty * b + b)) for c in range(tx * b, min(side, tx * b + b))]
        dev.onTileWeightsChanged(tx, ty, [(q, int(rng.integers(1, 50))) for q in box], gm)
        assert new.build(grid, weights=gm.weights)
        assert dev.stateDigest() == new.stateDigest()
        if gm.weights.max() < 60000:
            assert np.array_equal(dev.queryAllPairs(vps, gm), _weighted_distances(grid, gm.weights, vps))
