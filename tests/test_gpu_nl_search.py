"""The block-per-cell list search at its edges against the oracle's pairs,
bit for bit: pairs at exactly the list radius, atoms within 1e-10 A of each
other, shuffled and unwrapped atoms, atoms thousands of boxes away, a skewed
cell, four cells on an axis (the exact rows), more candidates than a block
ranks, cells without atoms, a batch of all kinds, and structures of more
atoms than the ranked index range holds, in and out of lattice order.  With and without
staging rows the list is the same.
"""
import numpy as np
import pytest
import torch

import oracle
from conftest import FCC, cubic, strained
from test_gpu_nl_rebuild import _build

pytestmark = pytest.mark.gpu

ak = pytest.importorskip("akitsushima_b200")
from akitsushima_b200 import _lib  # noqa: E402
from akitsushima_b200.neighbourlist import DeviceNeighbourList  # noqa: E402

R = 6.1


def _structure(name):
    rng = np.random.default_rng(3)
    if name == "ties":
        lat, pos, _ = cubic(FCC, R / np.sqrt(3.0), 10, ["Cu"] * 4, rattle=0.0, seed=1)
        return lat, pos
    if name == "dense":
        lat, pos, _ = cubic(FCC, 2.2, 14, ["Cu"] * 4, rattle=0.05, seed=2)
        return lat, pos
    cells = {"four": 8, "skewed": 10}.get(name, 9)
    lat, pos, _ = cubic(FCC, 3.58, cells, ["Cu"] * 4, rattle=0.08, seed=4)
    if name == "close":
        pos[1::7] = pos[0::7][:len(pos[1::7])] + rng.normal(size=(len(pos[1::7]), 3)) * 10.0 ** rng.integers(
            -13, -1, (len(pos[1::7]), 1))
    if name == "shuffled":
        pos = pos[rng.permutation(len(pos))] + rng.integers(-3, 4, (len(pos), 3)) @ lat
    if name == "far":
        pos[17] += 5000.0 * lat[1]
        pos[900] -= 6000.0 * lat[0]
    if name == "skewed":
        lat, pos = strained(lat, pos, 0.04, 6)
        shear = np.eye(3)
        shear[1, 0], shear[2, 0], shear[2, 1] = 0.3, -0.25, 0.2
        lat, pos = lat @ shear, pos @ shear
    if name == "hollow":
        pos = pos[(np.abs(pos - lat.diagonal() / 2) > 9.0).any(axis=1)]
    return lat, pos


NAMES = ["ties", "dense", "four", "close", "shuffled", "far", "skewed", "hollow"]


def _check(structs):
    batch = ak.Batch([s[0] for s in structs], [s[1] for s in structs], [np.zeros(len(s[1]), np.int32) for s in structs],
                     device="cuda")
    d = DeviceNeighbourList(R).build(batch)
    grids, n_cells = d._grid_table(batch)
    assert batch.n_atoms >= 10 * n_cells           # the block search
    i, j = (t.cpu().numpy() for t in d.half_pairs())
    want_i, want_j, base = [], [], 0
    for lat, pos in structs:
        oi, oj, _, _ = oracle.nl_build(lat, pos, R - 0.3, 0.3)
        want_i.append(oi + base)
        want_j.append(oj + base)
        base += len(pos)
    np.testing.assert_array_equal(i, np.concatenate(want_i))
    np.testing.assert_array_equal(j, np.concatenate(want_j))
    n, ns = batch.n_atoms, d.n_slots
    plain = int(_lib.lib().mbf_nl_workspace_bytes(n, n_cells))
    out = _build(batch, R, torch.as_tensor(grids, device="cuda"), n_cells, plain, ns)
    for got, ref in zip(out, (d.row_off[:n + 1], d.upper[:n], d.nbr[:ns], d.rev[:ns])):
        np.testing.assert_array_equal(got, ref.cpu().numpy())
    assert out[4] == d.max_row


@pytest.mark.parametrize("name", NAMES)
def test_block_search_gives_the_oracles_pairs(cuda_device, name):
    _check([_structure(name)])


def test_block_search_of_a_batch(cuda_device):
    _check([_structure(n) for n in NAMES])


@pytest.mark.parametrize("order", ["lattice", "axes_reversed", "rotated", "shuffled"])
def test_block_search_over_a_long_index(cuda_device, order):
    lat, pos, _ = cubic(FCC, 3.58, 33, ["Cu"] * 4, rattle=0.08, seed=7)
    assert len(pos) > 1 << 17
    if order == "axes_reversed":
        pos = np.ascontiguousarray(pos[:, ::-1])
    if order == "rotated":
        pos = np.roll(pos, 50001, axis=0)
    if order == "shuffled":
        pos = pos[np.random.default_rng(8).permutation(len(pos))]
    _check([(lat, pos)])
