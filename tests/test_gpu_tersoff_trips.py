"""The persistent blocks of the Tersoff centre kernel over three trips and more
(each takes its next centres while the last ones' rows are still in shared
memory): every staging bound, tables in shared memory and beyond it, with and
without lambda3, and every lane-group width.  Batches of three small
structures, repeated, each copy against the oracle.

Tolerances as test_gpu_tersoff_center: float64 1e-10 eV/atom and 1e-8 eV/A,
mixed 1e-6 eV/atom and 1e-5 eV/A scaled with the largest force.
"""
import numpy as np
import pytest
import torch

import oracle
from conftest import DIAMOND, cubic
from test_gpu_tersoff_center import _records

pytestmark = pytest.mark.gpu

ak = pytest.importorskip("akitsushima_b200")

# At most 148 SMs x 2048 threads are resident, a block has 64 threads or more,
# and takes 256 / (rows staged) centres: one trip is at most 4736 times that.
PER_TRIP = {32: 8 * 4736, 64: 4 * 4736, 128: 2 * 4736}
CASES = {
    # name: (species, record options, lattice constant, cells, list radius, row bound)
    "plain_row32": (1, {}, 5.431, 3, 4.0, 32),
    "records_row32": (3, dict(drop=5), 5.1, 3, 3.3, 32),
    "five_species_row32": (5, dict(lam=1.1), 5.1, 3, 3.3, 32),
    "plain_row64": (2, dict(same=True), 5.431, 3, 5.9, 64),
    "lambda3_row64": (4, dict(lam=0.4, m=1.0), 5.431, 3, 5.9, 64),
    "records_row128": (2, {}, 5.431, 4, 8.0, 128),
    "five_species_row128": (5, {}, 5.431, 4, 8.0, 128),
}


@pytest.mark.parametrize("lanes", [4, 8, 16])
@pytest.mark.parametrize("name", list(CASES))
def test_three_trips_match_oracle(cuda_device, name, lanes):
    ns, opts, a, cells, r_list, bound = CASES[name]
    sp, rec = _records(ns, 3, **opts)
    pot = ak.TersoffPotential(rec, species=sp)
    pot.lanes_per_atom = lanes
    structs, refs = [], []
    for k in range(3):
        lat, pos, _ = cubic(DIAMOND, a, cells, ["X0"] * 8, rattle=0.08, seed=4 + k)
        pos = pos[:len(pos) - 2 * k - 1]
        ids = np.random.default_rng(5 + k).integers(0, ns, len(pos)).astype(np.int32)
        i, j = oracle.nl_build(lat, pos, pot.r_cut, 0.02)[:2]
        structs.append((lat, pos, ids))
        refs.append(oracle.tersoff_multi(rec, sp, lat, pos, [sp[q] for q in ids], (i, j)))
    n = sum(len(s[1]) for s in structs)
    # a block's 21 KB or more of shared memory leave a third of that resident
    copies = -(-3 * PER_TRIP[bound] // (3 * n))
    batch = ak.Batch([s[0] for s in structs] * copies, [s[1] for s in structs] * copies,
                     [s[2] for s in structs] * copies, device=cuda_device)
    dl = ak.DeviceNeighbourList(max(r_list, pot.r_cut)).build(batch)
    assert bound // 2 * (bound > 32) < dl.max_row <= bound
    f0 = torch.as_tensor(np.concatenate([r[1] for r in refs]), device=cuda_device)
    e0 = torch.as_tensor(np.array([r[0] for r in refs]), device=cuda_device)
    top = max(1.0, float(f0.abs().max()))
    for prec, te, tf in (("fp64", 1e-10, 1e-8), ("mixed", 1e-6, 1e-5)):
        r = pot.evaluate(batch, dl, precision=prec)
        pot.status()
        de = (r.energy.view(copies, 3) - e0).abs() / torch.tensor([len(s[1]) for s in structs], device=cuda_device)
        assert float(de.max()) < te * max(1.0, float(e0.abs().max()) / n * 3)
        assert float((r.forces.view(copies, n, 3) - f0).abs().max()) < tf * top


def test_sw_row_bounds_are_the_ones_named(cuda_device):
    """The list radii of test_gpu_sw_center reach its three staging bounds."""
    from test_gpu_sw_center import CASES as SW
    for name, lo, hi in (("si_row32", 1, 32), ("si_row64", 33, 64), ("gesn_row128", 65, 128)):
        _, a, cells, r_list, _ = SW[name]
        lat, pos, _ = cubic(DIAMOND, a, cells, ["x"] * 8, rattle=0.1, seed=4)
        dl = ak.DeviceNeighbourList(r_list).build(ak.Batch.single(lat, pos, np.zeros(len(pos), np.int32),
                                                                  device=cuda_device))
        assert lo <= dl.max_row <= hi
