"""The Stillinger-Weber centre kernel at the edges of its dispatch, against
the oracle: row bounds (32, 64, 128 staged entries), more legs than a round of
lanes, tables in shared memory (up to three species) and beyond it, pairs of
different reach, published and general exponents, and every lane-group width.

Tolerances as tests/test_gpu_parity.py: float64 1e-10 eV/atom and 1e-8 eV/A,
mixed 1e-6 eV/atom and 1e-5 eV/A of ordinary bond lengths, scaled with the
largest force of the compressed cells.
"""
import numpy as np
import pytest

import oracle
from conftest import DIAMOND, SW_GESN, SW_SI, cubic, nested_records, strained

pytestmark = pytest.mark.gpu

ak = pytest.importorskip("akitsushima_b200")


def _records(ns, seed):
    """Records of ns species: symmetric pairs of different sigma and cutoff,
    lambda and cos0 per (i, j, k), general p and q."""
    rng = np.random.default_rng(seed)
    sp = [f"Y{k}" for k in range(ns)]
    pair = {}
    for a in range(ns):
        for b in range(a, ns):
            pair[a, b] = pair[b, a] = dict(epsilon=2.1 + 0.2 * rng.normal(), sigma=2.05 + 0.1 * rng.uniform(),
                                           a=1.7 + 0.15 * rng.uniform(), gamma=1.2 + 0.1 * rng.normal(), A=7.0, B=0.6,
                                           p=3.7 + 0.5 * rng.uniform(), q=0.4 * rng.uniform())
    out = {}
    for a in range(ns):
        for b in range(ns):
            for c in range(ns):
                rec = dict(pair[a, b] if b == c else pair[a, b], **{"lambda": 21.0 * rng.uniform(0.9, 1.1),
                                                                    "costheta0": -1 / 3 + 0.05 * rng.normal()})
                out[sp[a], sp[b], sp[c]] = rec
    return sp, out


CASES = {
    # name: (records, lattice constant, cells, list radius, strain)
    "si_row32": ("si", 5.431, 3, 4.1, 0.0),
    "si_row64": ("si", 5.431, 3, 5.9, 0.01),
    "gesn_row128": ("gesn", 5.762, 4, 8.3, 0.0),
    "gesn": ("gesn", 5.762, 3, 4.8, 0.0),
    "many_legs": ("gesn", 4.9, 3, 4.6, 0.0),
    "three": (3, 5.3, 3, 4.2, 0.0),
    "four": (4, 5.3, 3, 4.2, 0.01),
    "two_cells": ("si", 5.431, 2, 3.8, 0.0),
}


@pytest.mark.parametrize("lanes", [4, 8, 16])
@pytest.mark.parametrize("name", list(CASES))
def test_sw_center_matches_oracle(cuda_device, name, lanes):
    kind, a, cells, r_list, amp = CASES[name]
    lat, pos, _ = cubic(DIAMOND, a, cells, ["x"] * 8, rattle=0.1, seed=4)
    if amp:
        lat, pos = strained(lat, pos, amp, 5)
    keep = np.ones(len(pos), bool)
    keep[[1, 5]] = False                        # an atom count no group size divides
    pos = pos[keep]
    if kind == "si":
        sp, pot = ["Si"], ak.StillingerWeberPotential(SW_SI, species=["Si"])
    elif kind == "gesn":
        sp, pot = ["Ge", "Sn"], ak.StillingerWeberPotential(SW_GESN, species=["Ge", "Sn"])
    else:
        sp, rec = _records(kind, 3)
        pot = ak.StillingerWeberPotential(rec, species=sp)
    ids = np.random.default_rng(6).integers(0, len(sp), len(pos)).astype(np.int32)
    types = [sp[k] for k in ids]
    pot.lanes_per_atom = lanes
    batch = ak.Batch.single(lat, pos, ids, device=cuda_device)
    dl = ak.DeviceNeighbourList(max(r_list, pot.r_cut)).build(batch)
    i, j = oracle.nl_build(lat, pos, pot.r_cut, 0.02)[:2]
    if kind == "si":
        e0, f0, s0 = oracle.sw_single(SW_SI, lat, pos, (i, j))
    else:
        e0, f0, s0 = oracle.sw_multi(nested_records(SW_GESN) if kind == "gesn" else rec, sp, lat, pos, types, (i, j))
    vol = abs(np.linalg.det(lat))
    top = max(1.0, np.abs(f0).max())
    for prec, te, tf in (("fp64", 1e-10, 1e-8), ("mixed", 1e-6, 1e-5)):
        r = pot.evaluate(batch, dl, precision=prec)
        pot.status()
        assert abs(float(r.energy[0]) - e0) / len(pos) < te * max(1.0, abs(e0) / len(pos))
        assert np.abs(r.forces.cpu().numpy() - f0).max() < tf * top
        assert np.abs(r.virial.cpu().numpy().reshape(3, 3) / vol - s0).max() < tf * top


@pytest.mark.parametrize("pot", ["sw", "tersoff"])
def test_bad_list_entries_are_reported_and_skipped(cuda_device, pot):
    """A list entry, a reverse slot and a species outside their arrays: the
    evaluation reads and writes inside its arrays and the status says so."""
    lat, pos, types = cubic(DIAMOND, 5.431, 3, ["Si"] * 8, rattle=0.05, seed=6)
    p = ak.StillingerWeberPotential(SW_SI, species=["Si"]) if pot == "sw" else \
        ak.TersoffPotential(ak.TERSOFF_SI_1988, species=["Si"])
    for what in ("nbr", "rev", "types"):
        batch = ak.Batch.single(lat, pos, np.zeros(len(pos), np.int32), device=cuda_device)
        dl = ak.DeviceNeighbourList(4.1).build(batch)
        if what == "types":
            batch.types[7] = 3
        else:
            getattr(dl, what)[11] = 1 << 30
        p.evaluate(batch, dl)
        with pytest.raises(RuntimeError, match="device check failed"):
            p.status()
