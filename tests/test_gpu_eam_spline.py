"""setfl splines through the packed-table path and around its rule, against
the oracle: one to four species, r * phi and phi tables, tables that end
inside the cutoff (extrapolated), a grid that does not start at zero, every
lane width, diagonal and triclinic cells; and tables that keep the generic
path (different grids, non-uniform knots, a list shorter than the tables).

Tolerances as tests/test_gpu_parity.py: float64 1e-10 eV/atom and 1e-8 eV/A,
mixed 1e-6 eV/atom and 1e-5 eV/A.
"""
import numpy as np
import pytest

import oracle
from conftest import FCC, cubic, strained

pytestmark = pytest.mark.gpu

ak = pytest.importorskip("akitsushima_b200")
from akitsushima_b200.eam import EAMPotential, SpecFunction  # noqa: E402
from akitsushima_b200.published_parameters import ZHOU_2004  # noqa: E402


def _tables(species, n=1500, r0=0.0, r_end=None, over_r=True, uniform=True, second_n=None):
    """A spline EAMPotential of the Zhou alloy on grids of n knots."""
    from scipy.interpolate import CubicSpline
    pot = ak.zhou_eam({s: ZHOU_2004[s] for s in species}, species)
    end = pot.r_cut if r_end is None else r_end

    def grid(m):
        g = np.linspace(r0, end, m)
        return g if uniform else r0 + (end - r0) * np.linspace(0.0, 1.0, m) ** 1.05

    def fn(x, y, kind):
        cs = CubicSpline(x, y)
        return SpecFunction((kind, np.asarray(cs.x, float), np.asarray(cs.c, float)))

    r_g = grid(n)
    r_h = r_g if second_n is None else grid(second_n)
    pos = lambda g: np.where(g > 0.0, g, g[1])  # noqa: E731
    rho_g = np.linspace(0.0, 120.0, 800)
    F = {s: fn(rho_g, pot._F[s](rho_g), "spline") for s in species}
    rho = {s: fn(r_h, pot._rho[s](pos(r_h)), "spline") for s in species}
    phi = {k: fn(r_g, (r_g if over_r else 1.0) * f(pos(r_g)), "spline_over_r" if over_r else "spline")
           for k, f in pot._phi.items()}
    return EAMPotential(F, rho, phi, r_cut=pot.r_cut, species=species)


def _oracle(pot, lat, pos, types):
    sp = pot.species
    ns = len(sp)
    specs = [pot.rho_spec[s] for s in sp] + [pot.F_spec[s] for s in sp]
    fid = np.zeros((ns, ns), int)
    for a in range(ns):
        for b in range(a, ns):
            fid[a, b] = fid[b, a] = len(specs)
            specs.append(pot.phi_spec[frozenset((sp[a], sp[b]))])
    spec = oracle.EAMSpec(sp, specs, list(range(ns)), list(range(ns, 2 * ns)), fid, pot.r_cut)
    i, j = oracle.nl_build(lat, pos, pot.r_cut, 0.02)[:2]
    return oracle.eam(spec, lat, pos, types, (i, j))


CASES = {
    # name: (species, table options, cells, strain, lanes)
    "one": (["Ni"], {}, 4, 0.0, 4),
    "two_box": (["Cu", "Ni"], {}, 5, 0.0, 1),
    "two_triclinic": (["Cu", "Ni"], {}, 5, 0.015, 8),
    "phi_not_over_r": (["Cu", "Ni"], dict(over_r=False), 5, 0.0, 2),
    "grid_from_1A": (["Cu", "Ni"], dict(r0=1.0), 5, 0.0, 4),
    "ends_inside_cutoff": (["Ni"], dict(r0=2.2, r_end=5.2), 5, 0.0, 4),
    "below_first_knot": (["Ni"], dict(r0=2.6), 5, 0.0, 4),
    "four": (["Cu", "Ni", "Ag", "Pd"], dict(n=400), 5, 0.01, 4),
    "two_knots": (["Ni"], dict(n=4, r0=2.0), 4, 0.0, 4),
    # the generic path
    "grids_differ": (["Cu", "Ni"], dict(second_n=1400), 5, 0.0, 4),
    "knots_not_uniform": (["Cu", "Ni"], dict(uniform=False), 5, 0.0, 4),
    "tables_longer_than_list": (["Ni"], dict(n=20000), 4, 0.0, 4),
}


@pytest.mark.parametrize("name", list(CASES))
def test_spline_eam_matches_oracle(cuda_device, name):
    species, opts, n, amp, lanes = CASES[name]
    pot = _tables(species, **opts)
    pot.lanes_per_atom = lanes
    lat, pos, _ = cubic(FCC, 3.65, n, ["X"] * 4, rattle=0.06, seed=2)
    if amp:
        lat, pos = strained(lat, pos, amp, 3)
    pos = pos[:-1]
    ids = np.random.default_rng(4).integers(0, len(species), len(pos)).astype(np.int32)
    types = [species[k] for k in ids]
    e0, f0, s0 = _oracle(pot, lat, pos, types)
    batch = ak.Batch.single(lat, pos, ids, device=cuda_device)
    dl = ak.DeviceNeighbourList(pot.r_cut + 0.2).build(batch)
    vol = abs(np.linalg.det(lat))
    top = max(1.0, np.abs(f0).max())
    for prec, te, tf in (("fp64", 1e-10, 1e-8), ("mixed", 1e-6, 1e-5)):
        r = pot.evaluate(batch, dl, precision=prec)
        pot.status()
        assert abs(float(r.energy[0]) - e0) / len(pos) < te * max(1.0, abs(e0) / len(pos))
        assert np.abs(r.forces.cpu().numpy() - f0).max() < tf * top
        assert np.abs(r.virial.cpu().numpy().reshape(3, 3) / vol - s0).max() < tf * top


def test_halves_and_sites_use_the_tables(cuda_device):
    """The evaluation in two halves and the site terms give the whole call's
    values (the packed tables are rebuilt by each entry)."""
    pot = _tables(["Cu", "Ni"])
    lat, pos, _ = cubic(FCC, 3.65, 5, ["X"] * 4, rattle=0.06, seed=2)
    ids = np.random.default_rng(4).integers(0, 2, len(pos)).astype(np.int32)
    batch = ak.Batch.single(lat, pos, ids, device=cuda_device)
    dl = ak.DeviceNeighbourList(pot.r_cut + 0.2).build(batch)
    whole = pot.evaluate(batch, dl)
    e, f = whole.energy.clone(), whole.forces.clone()
    fp = pot.embedding(batch, dl)
    half = pot.forces_from_embedding(batch, dl, fp)
    assert abs(float(half.energy[0] - e[0])) < 1e-12 * abs(float(e[0]))
    assert float((half.forces - f).abs().max()) < 1e-12
    r, site_e, _, _ = pot.evaluate_sites(batch, dl)
    assert abs(float(site_e.sum() - e[0])) < 1e-10 * len(pos)
    assert float((r.forces - f).abs().max()) < 1e-12
