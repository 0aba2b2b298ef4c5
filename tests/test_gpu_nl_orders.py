"""Which cells the block search is given, against the oracle's pairs bit for
bit: structures of more atoms than its index map reaches whose numbering runs
by species (two species: every cell within reach; eight: some cells; in no
order: none), structures on both sides of five cells on an axis, and batches
whose structures have few cells on average, with and without one that has
many."""
import numpy as np
import pytest

import oracle
from conftest import FCC, cubic

pytestmark = pytest.mark.gpu

ak = pytest.importorskip("akitsushima_b200")
from akitsushima_b200.neighbourlist import DeviceNeighbourList  # noqa: E402


def _check(device, structs):
    batch = ak.Batch([s[0] for s in structs], [s[1] for s in structs],
                     [np.zeros(len(s[1]), np.int32) for s in structs], device=device)
    i, j = (t.cpu().numpy() for t in DeviceNeighbourList(6.1).build(batch).half_pairs())
    want, base = [], 0
    for lat, pos in structs:
        want.append(np.stack(oracle.nl_build(lat, pos, 5.8, 0.3)[:2]) + base)
        base += len(pos)
    want = np.concatenate(want, axis=1)
    np.testing.assert_array_equal(i, want[0])
    np.testing.assert_array_equal(j, want[1])


@pytest.mark.parametrize("species", [2, 3, 8])
def test_numbered_by_species(cuda_device, species):
    lat, pos, _ = cubic(FCC, 3.58, 33, ["Cu"] * 4, rattle=0.08, seed=7)
    kind = np.random.default_rng(1).integers(0, species, len(pos))
    _check(cuda_device, [(lat, pos[np.argsort(kind, kind="stable")])])


def _box(n, seed):
    lat, pos, _ = cubic(FCC, 3.58, n, ["Cu"] * 4, rattle=0.08, seed=seed)
    return lat, pos


@pytest.mark.parametrize("sizes", [(8,), (9,), (4, 6, 5), (4, 4, 4, 10), (9, 4), (10, 10, 4)])
def test_few_cells(cuda_device, sizes):
    _check(cuda_device, [_box(n, k) for k, n in enumerate(sizes)])


@pytest.mark.parametrize("axes", [(10, 8, 8), (8, 12, 9)])
def test_thin_boxes(cuda_device, axes):
    n = max(axes)
    lat, pos = _box(n, 3)
    keep = np.ones(len(pos), bool)
    cells = np.floor(np.repeat(np.indices((n, n, n)).reshape(3, -1).T, 4, axis=0))
    for k in range(3):
        keep &= cells[:, k] < axes[k]
    _check(cuda_device, [(np.diag(3.58 * np.array(axes)), pos[keep])])
