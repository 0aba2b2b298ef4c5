"""The block search's ranks over stencils whose atoms span many chunks of the
index (4096 indices each): repeated builds are the oracle's list, bit for bit."""
import numpy as np
import pytest

import oracle
from conftest import FCC, cubic

pytestmark = pytest.mark.gpu

ak = pytest.importorskip("akitsushima_b200")
from akitsushima_b200.neighbourlist import DeviceNeighbourList  # noqa: E402


@pytest.mark.parametrize("cells,shuffle", [(9, False), (12, True), (20, True), (28, True)])
def test_ranks_across_chunks(cuda_device, cells, shuffle):
    lat, pos, _ = cubic(FCC, 3.58, cells, ["Cu"] * 4, rattle=0.08, seed=11)
    if shuffle:
        pos = pos[np.random.default_rng(12).permutation(len(pos))]
    assert len(pos) <= 1 << 17
    oi, oj = oracle.nl_build(lat, pos, 5.8, 0.3)[:2]
    batch = ak.Batch.single(lat, pos, np.zeros(len(pos), np.int32), device=cuda_device)
    for _ in range(5):
        d = DeviceNeighbourList(6.1).build(batch)
        assert len(pos) >= 10 * d._grid_table(batch)[1]           # the block search
        i, j = (t.cpu().numpy() for t in d.half_pairs())
        np.testing.assert_array_equal(i, oi)
        np.testing.assert_array_equal(j, oj)
