"""Levels lifted viewpoint by viewpoint (the query kernel's chain units) against
the CPU restatement of the reference (tolerance 0), at the places where the route
changes: no level, some levels and all levels in the chain (viewpoint counts
on both sides of 4 per child), matrices on both sides of the padded order
1024, 768 columns (no power of two), one viewpoint, several in a leaf, in host and
device form and after an opening."""
import numpy as np
import pytest

from helpers import make_grid
from htrip_b200 import workloads as W
from oracle.ref import PortOracle, port_available, port_bfs

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not port_available(), reason="oracle port not built (make -C oracle port)")]

CASES = [
    # kind, rows, cols, b, g, viewpoint counts
    ("noise", 16, 16, 8, 2, (1, 2, 16, 17)),       # H = 1: the root itself in the chain, then not
    ("noise", 60, 52, 8, 2, (1, 5, 64, 65, 257)),  # H = 3
    ("street", 128, 120, 4, 2, (3, 16, 17, 256)),  # five levels, at most four in the chain
    ("maze", 97, 90, 12, 2, (2, 30, 200)),         # level 2 of padded order 768
    ("noise", 64, 64, 32, 2, (2, 16, 40)),         # level 1 of padded order 512
    ("noise", 64, 60, 4, 4, (4, 60, 700)),         # level 2 of padded order 1024
    ("noise", 40, 40, 5, 3, (3, 50)),
    ("open", 30, 30, 30, 2, (2, 9)),               # H = 0
]


@pytest.mark.parametrize("kind,rows,cols,b,g,ks", CASES)
def test_queries_match_the_oracle(gpu, kind, rows, cols, b, g, ks):
    import torch

    from htrip_b200.minplus_oracle import HierarchyConfig, MinPlusOracle
    truth = make_grid(kind, rows, cols, rows + b)
    observed, cells = W.withheld_open(truth, 20, 5)
    dev, cpu = MinPlusOracle(HierarchyConfig(b, g, g)), PortOracle(b, g)
    assert dev.build(observed) and cpu.build(observed)
    for step in range(2):
        for k in ks:
            free = W.sample_free(observed, k, k + step)
            vps = np.concatenate([free, free[: max(0, min(k - len(free), len(free)))]])  # repeats where cells run out
            got = dev.queryAllPairs(vps, observed)
            assert np.array_equal(got, cpu.query(vps, observed)), k
            assert np.array_equal(got, port_bfs(observed, vps)), k
            v = torch.from_numpy(np.ascontiguousarray(vps)).cuda()
            p = torch.ones(len(vps), dtype=torch.uint8, device="cuda")
            out = torch.empty((len(vps), len(vps)), dtype=torch.uint16, device="cuda")
            torch.cuda.synchronize()
            dev.queryAllPairsDevice(v.data_ptr(), p.data_ptr(), len(vps), out.data_ptr())
            dev.synchronize()
            assert np.array_equal(out.cpu().numpy(), got), k
        observed[cells[:, 0], cells[:, 1]] = W.FREE
        dev.onBatchCellsOpened(cells, observed)
        cpu.open_batch(cells, observed)


@pytest.mark.parametrize("rows,cols,b,g,k", [(64, 64, 8, 2, 300), (60, 57, 5, 3, 200), (64, 64, 4, 4, 500),
                                             (200, 200, 16, 2, 700)])
def test_seam_rows(gpu, rows, cols, b, g, k):
    """Winding corridors: the shortest way between two ports of a child runs inside it
    for some and outside for others.  Full and incremental queries, after openings."""
    from htrip_b200.minplus_oracle import HierarchyConfig, IncrementalState, MinPlusOracle
    truth = np.full((rows, cols), W.FREE, np.uint8)
    truth[1::2] = W.OBSTACLE
    for i in range(1, rows, 2):
        truth[i, cols - 1 if (i // 2) % 2 == 0 else 0] = W.FREE
        truth[i, (7 * i) % cols] = W.FREE
    observed, cells = W.withheld_open(truth, 30, 5)
    dev, cpu = MinPlusOracle(HierarchyConfig(b, g, g)), PortOracle(b, g)
    assert dev.build(observed) and cpu.build(observed)
    vps, state = W.sample_free(observed, k, 3), IncrementalState()
    for part in (cells[:0], cells[:1], cells[1:]):
        if len(part):
            observed[part[:, 0], part[:, 1]] = W.FREE
            dev.onBatchCellsOpened(part, observed)
            cpu.open_batch(part, observed)
        want = port_bfs(observed, vps)
        assert np.array_equal(cpu.query(vps, observed), want)
        assert np.array_equal(dev.queryAllPairs(vps, observed), want)
        assert np.array_equal(dev.queryAllPairsIncremental(vps, observed, state), want)
