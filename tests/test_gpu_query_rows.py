"""Operand rows of a query's project and meet items: all finite ports where nearly every
port lies on a seam (large groups), the seam ports elsewhere.  Against a breadth-first
search on the grid, tolerance 0, host-planned, device-planned and incremental, on both
sides of the rule (group 4 and 5, tile sides that move it)."""
import numpy as np
import pytest

from htrip_b200 import workloads as W
from oracle.ref import port_available, port_bfs

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not port_available(), reason="oracle port not built (make -C oracle port)")]


@pytest.mark.parametrize("rows,cols,b,g,k", [(128, 120, 8, 4, 300), (100, 97, 20, 5, 200), (50, 50, 2, 5, 90),
                                             (130, 128, 16, 8, 260), (64, 60, 8, 8, 70), (128, 128, 8, 16, 520),
                                             (16, 16, 4, 4, 60)])
def test_rows_by_group(gpu, rows, cols, b, g, k):
    import torch

    from htrip_b200.minplus_oracle import HierarchyConfig, IncrementalState, MinPlusOracle
    truth = np.full((rows, cols), W.FREE, np.uint8)
    truth[1::2] = W.OBSTACLE
    for i in range(1, rows, 2):
        truth[i, cols - 1 if (i // 2) % 2 == 0 else 0] = W.FREE
        truth[i, (7 * i) % cols] = W.FREE
    observed, cells = W.withheld_open(truth, 25, 5)
    dev, state = MinPlusOracle(HierarchyConfig(b, g, g)), IncrementalState()
    assert dev.build(observed)
    vps = np.ascontiguousarray(W.sample_free(observed, k, 3), dtype=np.int32)
    v, p = torch.from_numpy(vps).cuda(), torch.ones(len(vps), dtype=torch.uint8, device="cuda")
    out = torch.empty((len(vps), len(vps)), dtype=torch.uint16, device="cuda")
    for part in (cells[:0], cells[:1], cells[1:]):
        if len(part):
            observed[part[:, 0], part[:, 1]] = W.FREE
            dev.onBatchCellsOpened(part, observed)
        want = port_bfs(observed, vps)
        assert np.array_equal(dev.queryAllPairs(vps, observed), want)
        assert np.array_equal(dev.queryAllPairsIncremental(vps, observed, state), want)
        torch.cuda.synchronize()
        dev.queryAllPairsDevice(v.data_ptr(), p.data_ptr(), len(vps), out.data_ptr())
        dev.synchronize()
        assert np.array_equal(out.cpu().numpy(), want)
