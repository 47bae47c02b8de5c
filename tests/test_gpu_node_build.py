"""Node matrices made by contracting the seam edges (csrc/node_build.cu): every
leaf and node matrix after a build and after a blocked cell's rebuild against
the CPU restatement of the reference (tolerance 0), at the sizes where the
kernels change: nodes that fit one CTA and nodes that do not, one and several
rounds of 64 seams, ports per child on and off a tile's edge, distances below
and above half of the 16-bit range, no active seam at all, g other than 2."""
import numpy as np
import pytest

from helpers import FREE, OBST, make_grid
from htrip_b200 import workloads as W
from oracle.ref import PortOracle, port_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not port_available(), reason="oracle port not built (make -C oracle port)")]


def snake(rows, cols):
    """One corridor that fills the map: distances up to rows * cols / 2."""
    g = np.full((rows, cols), FREE, np.uint8)
    g[1::2] = OBST
    for i in range(1, rows, 2):
        g[i, cols - 1 if (i // 2) % 2 == 0 else 0] = FREE
    return g


GRIDS = {
    "open": lambda r, c: np.full((r, c), FREE, np.uint8),
    "shut": lambda r, c: np.full((r, c), OBST, np.uint8),
    "noise": lambda r, c: make_grid("noise", r, c, r + c),
    "street": lambda r, c: make_grid("street", r, c, r + c),
    "maze": lambda r, c: make_grid("maze", r, c, r + c),
    "snake": snake,
}

CASES = [
    # kind, rows, cols, b, g
    ("open", 32, 32, 16, 2),      # one small node (64 seams)
    ("open", 64, 64, 16, 2),      # its parent: two rounds, 128 seams all active
    ("open", 130, 128, 32, 2),    # 33-port overlap: general nodes from the leaves up
    ("shut", 70, 50, 8, 2),
    ("noise", 60, 40, 4, 2),
    ("noise", 75, 75, 5, 2),      # 16 ports per child
    ("noise", 70, 66, 17, 2),     # 64 ports per child, 68 seams
    ("noise", 80, 72, 18, 2),     # 68 ports per child
    ("noise", 54, 50, 3, 3),
    ("noise", 64, 60, 4, 4),
    ("noise", 50, 44, 2, 5),
    ("street", 120, 100, 8, 2),
    ("maze", 128, 97, 8, 2),
    ("snake", 64, 64, 8, 2),      # distances up to 2 k
    ("noise", 21, 20, 7, 2),      # leaves of 49 cells (fewer than their padded order)
    ("noise", 40, 36, 9, 2),      # leaves of 81 cells: 256 threads, padded order 128
    ("maze", 31, 31, 31, 2),      # one leaf of 961 cells, 32 sources a time
    ("snake", 200, 200, 16, 2),   # up to 20 k: sums above half of the range
]


def same_matrices(dev, cpu):
    for i in range(dev.num_leaf_tiles_x ** 2):
        assert np.array_equal(dev.leaf_D(i), cpu.leaf_D(i)), f"leaf {i}"
    for lvl in range(1, dev.H + 1):
        for n in range(dev.level_dims(lvl)[3]):
            assert np.array_equal(dev.node_DU(lvl, n), cpu.node_DU(lvl, n)), f"level {lvl} node {n}"


@pytest.mark.parametrize("kind,rows,cols,b,g", CASES)
def test_build_and_rebuild_match_the_oracle(gpu, kind, rows, cols, b, g):
    from htrip_b200.minplus_oracle import HierarchyConfig, MinPlusOracle
    grid = GRIDS[kind](rows, cols)
    dev, cpu = MinPlusOracle(HierarchyConfig(b, g, g)), PortOracle(b, g)
    assert dev.build(grid) and cpu.build(grid)
    same_matrices(dev, cpu)
    free = np.argwhere(grid == FREE)
    if len(free) == 0:
        return
    p = tuple(int(x) for x in free[len(free) // 3])
    grid[p] = OBST
    dev.onCellBlocked(p, grid)
    cpu = PortOracle(b, g)
    assert cpu.build(grid)
    same_matrices(dev, cpu)


@pytest.mark.parametrize("rows,cols,b,top", [(48, 40, 8, 9), (96, 96, 16, 400), (64, 64, 32, 3000)])
def test_weighted_build_matches_dijkstra(gpu, rows, cols, b, top):
    """Seam weights as incidence offsets, sums up to and beyond INF."""
    from scipy.sparse import coo_matrix
    from scipy.sparse.csgraph import dijkstra

    from htrip_b200.minplus_oracle import INF, GridMap, HierarchyConfig, MinPlusOracle
    grid = make_grid("noise", rows, cols, rows)
    wts = np.random.default_rng(b).integers(1, top + 1, size=grid.shape).astype(np.uint16)
    idx = np.arange(grid.size).reshape(grid.shape)
    ends, cost = [], []
    for a, c in ((np.s_[1:], np.s_[:-1]), (np.s_[:, 1:], np.s_[:, :-1])):
        ok = (grid[a] == FREE) & (grid[c] == FREE)
        ends.append(np.stack([idx[a][ok], idx[c][ok]]))
        cost.append(np.maximum(1, (wts[a][ok].astype(int) + wts[c][ok]) // 2))
    ends, cost = np.concatenate(ends, axis=1), np.concatenate(cost)
    graph = coo_matrix((cost, (ends[0], ends[1])), shape=(grid.size, grid.size)).tocsr()
    vps = W.sample_free(grid, 40, 7)
    at = idx[vps[:, 0], vps[:, 1]]
    want = np.minimum(dijkstra(graph, directed=False, indices=at)[:, at], INF).astype(np.uint16)
    dev = MinPlusOracle(HierarchyConfig(b, 2, 2))
    gm = GridMap(grid, wts)
    assert dev.build(gm)
    assert np.array_equal(dev.queryAllPairs(vps, gm), want)
