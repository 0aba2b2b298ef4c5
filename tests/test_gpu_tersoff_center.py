"""The Tersoff centre kernel at the edges of its dispatch, against the oracle:
row bounds (32, 64, 128 staged entries), bonds in several rounds of four
lanes, tables in shared memory (up to four species) and beyond it, records
that do and do not share their angular function, absent records, lambda3 with
either power, and every lane-group width.

Tolerances as tests/test_gpu_parity.py: float64 1e-10 eV/atom and 1e-8 eV/A,
mixed 1e-6 eV/atom and 1e-5 eV/A of ordinary bond lengths; the compressed
cells' forces are larger, so the float32 terms' bound scales with the largest
force.
"""
import numpy as np
import pytest

import oracle
from conftest import DIAMOND, cubic

pytestmark = pytest.mark.gpu

ak = pytest.importorskip("akitsushima_b200")


def _records(ns, seed, lam=0.0, m=3.0, same=False, drop=0):
    """(i, j, k) records of ns species: symmetric pair parameters around
    silicon's, angular parameters per record (or per centre with `same`)."""
    rng = np.random.default_rng(seed)
    sp = [f"X{k}" for k in range(ns)]
    pair, cen = {}, {}
    for a in range(ns):
        cen[a] = dict(c=100390.0 * rng.uniform(0.8, 1.2), d=16.217 * rng.uniform(0.8, 1.2), h=-0.6 + rng.uniform(-0.1, 0.1))
        for b in range(a, ns):
            u = rng.uniform(0.95, 1.05, 4)
            pair[a, b] = pair[b, a] = dict(A=1830.8 * u[0], B=471.18 * u[1], lambda1=2.4799 * u[2], lambda2=1.7322 * u[3],
                                           R=2.75 + rng.uniform(-0.1, 0.1), D=0.15)
    out = {}
    for a in range(ns):
        for b in range(ns):
            for c in range(ns):
                ang = dict(cen[a]) if same else dict(c=100390.0 * rng.uniform(0.8, 1.2), d=16.217 * rng.uniform(0.8, 1.2),
                                                     h=-0.6 + rng.uniform(-0.1, 0.1))
                rec = dict(ang, lambda3=lam, m=m, gamma=1.0 if same else rng.uniform(0.9, 1.1))
                if b == c:
                    rec.update(pair[a, b], beta=1.1e-6, n=0.78734)
                out[sp[a], sp[b], sp[c]] = rec
    for key in [k for k in out if k[1] != k[2]][:drop]:
        del out[key]
    return sp, out


CASES = {
    # name: (ns, record options, lattice constant, cells, list radius)
    "one_row32": (1, {}, 5.431, 3, 4.0),
    "plain_row64": (2, dict(same=True), 5.431, 3, 5.9),
    "records_row128": (2, dict(), 5.431, 4, 8.0),
    "dense_bonds": (2, dict(same=True), 3.9, 3, 3.3),
    "dense_records": (3, dict(drop=5), 3.9, 3, 3.3),
    "lambda3_m3": (2, dict(lam=1.3, m=3.0), 5.1, 3, 3.3),
    "lambda3_m1": (4, dict(lam=0.4, m=1.0), 5.1, 3, 3.3),
    "five_species": (5, dict(lam=1.1), 5.1, 3, 3.3),
    "two_cells": (1, {}, 5.431, 2, 3.0),
}


@pytest.mark.parametrize("lanes", [4, 8, 16])
@pytest.mark.parametrize("name", list(CASES))
def test_tersoff_center_matches_oracle(cuda_device, name, lanes):
    ns, opts, a, cells, r_list = CASES[name]
    sp, rec = _records(ns, 3, **opts)
    lat, pos, _ = cubic(DIAMOND, a, cells, ["X0"] * 8, rattle=0.08, seed=4)
    keep = np.ones(len(pos), bool)
    keep[[1, 5]] = False                        # an atom count no group size divides
    pos = pos[keep]
    ids = np.random.default_rng(5).integers(0, ns, len(pos)).astype(np.int32)
    types = [sp[k] for k in ids]
    pot = ak.TersoffPotential(rec, species=sp)
    pot.lanes_per_atom = lanes
    batch = ak.Batch.single(lat, pos, ids, device=cuda_device)
    dl = ak.DeviceNeighbourList(max(r_list, pot.r_cut)).build(batch)
    i, j = oracle.nl_build(lat, pos, pot.r_cut, 0.02)[:2]
    e0, f0, s0 = oracle.tersoff_multi(rec, sp, lat, pos, types, (i, j))
    vol = abs(np.linalg.det(lat))
    top = max(1.0, np.abs(f0).max())
    for prec, te, tf in (("fp64", 1e-10, 1e-8), ("mixed", 1e-6, 1e-5)):
        r = pot.evaluate(batch, dl, precision=prec)
        pot.status()
        assert abs(float(r.energy[0]) - e0) / len(pos) < te * max(1.0, abs(e0) / len(pos))
        assert np.abs(r.forces.cpu().numpy() - f0).max() < tf * top
        assert np.abs(r.virial.cpu().numpy().reshape(3, 3) / vol - s0).max() < tf * top


def test_row_bounds_are_the_ones_named(cuda_device):
    """The three list radii above reach the three staging bounds."""
    for name, lo, hi in (("one_row32", 1, 32), ("plain_row64", 33, 64), ("records_row128", 65, 128)):
        _, _, a, cells, r_list = CASES[name]
        lat, pos, _ = cubic(DIAMOND, a, cells, ["X0"] * 8, rattle=0.08, seed=4)
        dl = ak.DeviceNeighbourList(r_list).build(ak.Batch.single(lat, pos, np.zeros(len(pos), np.int32),
                                                                  device=cuda_device))
        assert lo <= dl.max_row <= hi


def test_row_longer_than_the_bound_is_reported(cuda_device):
    """A list whose stated longest row is too small: no force from such a
    row, and the status says so."""
    lat, pos, _ = cubic(DIAMOND, 5.431, 3, ["X0"] * 8, rattle=0.05, seed=6)
    sp, rec = _records(1, 3)
    pot = ak.TersoffPotential(rec, species=sp)
    batch = ak.Batch.single(lat, pos, np.zeros(len(pos), np.int32), device=cuda_device)
    dl = ak.DeviceNeighbourList(5.9).build(batch)
    dl.max_row = 32
    pot.evaluate(batch, dl)
    with pytest.raises(RuntimeError, match="device check failed"):
        pot.status()
