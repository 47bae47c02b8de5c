"""Closures of an opening (csrc/open.cu, closure.cuh) against the CPU restatement
of the reference (every matrix and the statistics, tolerance 0), at the places where
they change: matrices of padded order 64, 128 and more, pivot counts around a
step of 16 and a round of 64, one and several rounds, distances below and above
half of the 16-bit range (where the clamped form takes over, also after the half
range turned out too small)."""
import numpy as np
import pytest

from helpers import FREE, OBST, UNK, make_grid
from htrip_b200 import workloads as W
from oracle.ref import PortOracle, port_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not port_available(), reason="oracle port not built (make -C oracle port)")]


def snake(rows, cols):
    g = np.full((rows, cols), FREE, np.uint8)
    g[1::2] = OBST
    for i in range(1, rows, 2):
        g[i, cols - 1 if (i // 2) % 2 == 0 else 0] = FREE
    return g


CASES = [
    # kind, rows, cols, b, g, cells opened per call
    ("noise", 32, 32, 8, 2, (1, 2, 14, 40)),      # orders 64, 128, 256
    ("open", 64, 64, 8, 2, (16, 17, 300)),
    ("noise", 48, 48, 4, 2, (5, 120)),
    ("street", 128, 120, 8, 2, (64, 400)),
    ("noise", 64, 64, 16, 2, (3, 200)),           # leaves of order 256
    ("noise", 60, 60, 5, 3, (7, 90)),
    ("maze", 128, 128, 8, 2, (9, 250)),
    ("snake", 64, 64, 8, 2, (40, 160)),           # distances up to 2 k
    ("snake", 200, 200, 16, 2, (80, 200)),        # up to 20 k
]


@pytest.mark.parametrize("kind,rows,cols,b,g,steps", CASES)
def test_openings_match_the_oracle(gpu, kind, rows, cols, b, g, steps):
    from htrip_b200.minplus_oracle import HierarchyConfig, MinPlusOracle
    truth = snake(rows, cols) if kind == "snake" else make_grid(kind, rows, cols, rows + b)
    observed, cells = W.withheld_open(truth, sum(steps), 11)
    dev, cpu = MinPlusOracle(HierarchyConfig(b, g, g)), PortOracle(b, g)
    assert dev.build(observed) and cpu.build(observed)
    at = 0
    for m in steps:
        part = cells[at:at + m]
        at += m
        if len(part) == 0:
            break
        assert (observed[part[:, 0], part[:, 1]] == UNK).all()
        observed[part[:, 0], part[:, 1]] = FREE
        dev.onBatchCellsOpened(part, observed)
        cpu.open_batch(part, observed)
        st = dev.last_batch_stats
        assert (st.n_touched_leaves, st.n_dirty_ancestors, st.n_pivots) == cpu.stats()
        for i in range(dev.num_leaf_tiles_x ** 2):
            assert np.array_equal(dev.leaf_D(i), cpu.leaf_D(i)), f"leaf {i}"
        for lvl in range(1, dev.H + 1):
            for n in range(dev.level_dims(lvl)[3]):
                assert np.array_equal(dev.node_DU(lvl, n), cpu.node_DU(lvl, n)), f"level {lvl} node {n}"


@pytest.mark.parametrize("maps", [
    ((64, 8, 2), (64, 16, 2)),
    ((32, 4, 2), (200, 8, 2), (60, 5, 3)),                # the third launch runs by itself
    ((32, 8, 2), (256, 16, 2), (48, 16, 2), (48, 4, 2), (32, 8, 2)),
])
def test_launches_side_by_side(gpu, maps):
    """One opening over indexes of several (b, g): their launches share the GPU."""
    from htrip_b200.minplus_oracle import Batch, HierarchyConfig, MinPlusOracle
    batch, runs = Batch(), []
    for i, (side, b, g) in enumerate(maps):
        observed, cells = W.withheld_open(make_grid("noise", side, side, i), 60, i)
        dev, cpu = MinPlusOracle(HierarchyConfig(b, g, g)), PortOracle(b, g)
        assert dev.build(observed) and cpu.build(observed)
        runs.append((dev, cpu, observed, cells))
    for at, m in ((0, 3), (3, 57)):
        parts = [cells[at:at + m] for _, _, _, cells in runs]
        for (dev, cpu, observed, _), part in zip(runs, parts):
            observed[part[:, 0], part[:, 1]] = FREE
        batch.open([(dev, part, observed) for (dev, _, observed, _), part in zip(runs, parts)])
        for (dev, cpu, observed, _), part in zip(runs, parts):
            cpu.open_batch(part, observed)
            st = dev.last_batch_stats
            assert (st.n_touched_leaves, st.n_dirty_ancestors, st.n_pivots) == cpu.stats()
            for i in range(dev.num_leaf_tiles_x ** 2):
                assert np.array_equal(dev.leaf_D(i), cpu.leaf_D(i)), f"leaf {i}"
            for lvl in range(1, dev.H + 1):
                for n in range(dev.level_dims(lvl)[3]):
                    assert np.array_equal(dev.node_DU(lvl, n), cpu.node_DU(lvl, n)), f"level {lvl} node {n}"
