"""Mixed precision is as accurate as its float32 terms allow: isolated pairs
over the whole range of distances, site energies against the float64
evaluation's."""
import numpy as np
import pytest

from conftest import FCC, SW_SI, cubic

pytestmark = pytest.mark.gpu

ak = pytest.importorskip("akitsushima_b200")
from akitsushima_b200 import eam  # noqa: E402
from akitsushima_b200.published_parameters import ZHOU_2004  # noqa: E402


def _dimers(lo, hi, n=24, seed=3):
    """n^3 pairs, 12 A apart, of distances spread evenly over (lo, hi) in
    random directions: (lattice, positions, distances)."""
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3) * 12.0
    r = np.linspace(lo, hi, len(g) + 2)[1:-1]
    u = rng.normal(size=g.shape)
    u /= np.linalg.norm(u, axis=1)[:, None]
    return np.eye(3) * 12.0 * n, np.concatenate([g, g + u * r[:, None]]), r


def _site_energies(pot, lat, pos, device):
    batch = ak.Batch.single(lat, pos, np.zeros(len(pos), np.int32), device=device)
    dl = ak.DeviceNeighbourList(pot.r_cut + 0.3).build(batch)
    out = {}
    for prec in ("mixed", "fp64"):
        out[prec] = pot.evaluate_sites(batch, dl, precision=prec)[1].cpu().numpy().copy()
        pot.status()
    return out["mixed"], out["fp64"]


def test_tersoff_two_body_terms_are_float64(cuda_device):
    """A pair alone has no zeta term, so its energy is the two-body part with
    bond order 1, float64 in both precisions: the same operations on the same
    distance.  2e-15 of the energy scale allows for a compiler's different
    contraction."""
    pot = ak.TersoffPotential(ak.TERSOFF_SI_1988, species=["Si"])
    lat, pos, _ = _dimers(1.9, pot.r_cut)
    mixed, fp64 = _site_energies(pot, lat, pos, cuda_device)
    assert np.abs(fp64).max() > 0.5
    assert np.abs(mixed - fp64).max() <= 2e-15 * np.abs(fp64).max()


def test_sw_pair_term_rounds_its_power_once(cuda_device):
    """The float32 pair term of silicon (p = 4) errs as its formula does in
    float32 with x^-4 rounded once, emulated here: the same rms over 13,824
    distances.  The rms of so many has a spread of 0.6 %; 1.5 % is allowed.
    x^-4 from 1 / x by two squarings errs 3.4 % more."""
    f = np.float32
    pot = ak.StillingerWeberPotential(SW_SI, species=["Si"])
    lat, pos, r = _dimers(2.0, 3.6)
    mixed, fp64 = _site_energies(pot, lat, pos, cuda_device)
    n = len(r)
    e = mixed[:n] + mixed[n:]
    np.testing.assert_allclose(fp64[:n], fp64[n:], rtol=1e-12)
    eps, sig, a, A, B = (f(SW_SI[k]) for k in ("epsilon", "sigma", "a", "A", "B"))
    x = r.astype(f) / sig
    ex = np.exp((f(1) / (x - a)).astype(float)).astype(f)
    emulated = eps * A * ex * (B * (x.astype(float) ** -4).astype(f) - f(1))
    exact = 2.0 * fp64[:n]
    rms = lambda v: np.sqrt(np.mean((v - exact) ** 2))  # noqa: E731
    assert rms(e) <= 1.015 * rms(emulated)


def test_setfl_energy_has_no_bias(cuda_device):
    """Each pair's float32 value errs by parts of 1e-7 of tenths of an eV in
    either direction, so over 4000 atoms of about 40 pairs each the mean
    energy error averages to some 1e-9 eV an atom (3e-9 measured with a
    float64 1 / r); an inverse distance that errs to one side leaves 2e-8."""
    lat, pos, _ = cubic(FCC, 3.58, 10, ["x"] * 4, rattle=0.08, seed=1)
    ids = np.random.default_rng(6).integers(0, 2, len(pos)).astype(np.int32)
    pot = eam.tabulate(ak.zhou_eam({s: ZHOU_2004[s] for s in ("Cu", "Ni")}, ["Cu", "Ni"]))
    batch = ak.Batch.single(lat, pos, ids, device=cuda_device)
    dl = ak.DeviceNeighbourList(pot.r_cut + 0.3).build(batch)
    e = {p: float(pot.evaluate(batch, dl, precision=p).energy[0]) for p in ("mixed", "fp64")}
    pot.status()
    assert abs(e["mixed"] - e["fp64"]) < 1e-8 * len(pos)
