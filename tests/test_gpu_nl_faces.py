"""The block search of atoms on cell faces and on the box's own faces: perfect
fcc crystals under strain, whose atoms lie on integer fractions up to the
rounding of the lattice product, each also shifted by a few units in the last
place to either side of the face and by whole boxes; the oracle's pairs, bit
for bit."""
import numpy as np
import pytest

import oracle
from conftest import FCC, cubic

pytestmark = pytest.mark.gpu

ak = pytest.importorskip("akitsushima_b200")
from akitsushima_b200.neighbourlist import DeviceNeighbourList  # noqa: E402

STRAINS = {
    "xy": [[0.0, 0.02, 0.0], [0.02, 0.0, 0.0], [0.0, 0.0, 0.0]],
    "full": [[0.013, 0.02, -0.011], [0.02, -0.007, 0.017], [-0.011, 0.017, 0.005]],
    "shear": [[0.0, 0.0, 0.0], [0.25, 0.0, 0.0], [-0.2, 0.15, 0.0]],
}


@pytest.mark.parametrize("ulps", [0, -2, 2, "mixed"])
@pytest.mark.parametrize("name", list(STRAINS))
def test_atoms_on_faces(cuda_device, name, ulps):
    lat, pos, _ = cubic(FCC, 3.58, 10, ["Ni"] * 4, rattle=0.0, seed=1)
    M = np.eye(3) + np.array(STRAINS[name])
    lat, pos = lat @ M, pos @ M
    rng = np.random.default_rng(2)
    k = rng.integers(-3, 4, pos.shape) if ulps == "mixed" else np.full(pos.shape, float(ulps))
    pos = pos + k * np.spacing(np.abs(pos).max())
    if ulps == "mixed":
        pos = pos + rng.integers(-2, 3, pos.shape) @ lat
    oi, oj = oracle.nl_build(lat, pos, 5.8, 0.3)[:2]
    batch = ak.Batch.single(lat, pos, np.zeros(len(pos), np.int32), device=cuda_device)
    d = DeviceNeighbourList(6.1).build(batch)
    assert len(pos) >= 10 * d._grid_table(batch)[1]           # the block search
    i, j = (t.cpu().numpy() for t in d.half_pairs())
    np.testing.assert_array_equal(i, oi)
    np.testing.assert_array_equal(j, oj)
