"""The allocation-free query takes what its fixed 64 MiB hold, whatever schedule the
lowest levels would use: requests whose plan fits only without the lowest levels'
per-viewpoint table."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,b,k", [(128, 4, 2911), (256, 8, 2544), (512, 8, 1936)])
def test_request_that_just_fits(gpu, side, b, k):
    from htrip_b200.minplus_oracle import HierarchyConfig, MinPlusOracle
    grid = np.ones((side, side), np.uint8)
    dev = MinPlusOracle(HierarchyConfig(b, 2, 2))
    assert dev.build(grid)
    i = np.arange(k)
    vps = np.stack([i % b, i // b % b], axis=1).astype(np.int32)  # all in one leaf
    got = dev.queryAllPairsNoAlloc(vps, grid)
    want = np.abs(vps[:, None, 0] - vps[None, :, 0]) + np.abs(vps[:, None, 1] - vps[None, :, 1])
    assert np.array_equal(got, want.astype(np.uint16))
