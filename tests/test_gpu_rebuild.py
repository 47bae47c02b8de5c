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
