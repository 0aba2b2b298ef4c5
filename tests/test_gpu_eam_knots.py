"""setfl tables whose knots are uniform only to the tolerance of the interval
guess: the offset within an interval comes from the knots themselves, as the
oracle's does.

Tolerance: a pair's distance carries the rounding of coordinates below 20 A
(1e-14 A) and the tables curve by tens of eV/A^2, so a force of about 80 pairs
is good to 1e-11 eV/A; 1e-10 of the largest force is asked.  The knots are up
to 1.3e-9 A off the uniform grid, a hundred times what that leaves.
"""
import numpy as np
import pytest

from conftest import FCC, cubic
from test_gpu_eam_spline import _oracle, _tables

ak = pytest.importorskip("akitsushima_b200")
from akitsushima_b200.eam import EAMPotential, SpecFunction  # noqa: E402


def _stretched(pot, amp):
    """pot's pair and density splines with knots moved by amp t (1 - t) of the
    range (their spacings differ by amp), the coefficients as they are."""
    def move(spec):
        x = np.asarray(spec[1])
        t = (x - x[0]) / (x[-1] - x[0])
        return SpecFunction((spec[0], x + amp * t * (1.0 - t) * (x[-1] - x[0]), spec[2]))

    return EAMPotential({s: SpecFunction(v) for s, v in pot.F_spec.items()},
                        {s: move(v) for s, v in pot.rho_spec.items()},
                        {tuple(k) if len(k) == 2 else (*k, *k): move(v) for k, v in pot.phi_spec.items()},
                        r_cut=pot.r_cut, species=pot.species)


@pytest.mark.parametrize("knots,flags", [("linspace", (1.0, 1.0)), ("multiples", (1.0, 1.0)), ("summed", None),
                                         ("stretched", (1.0, 0.0)), ("uneven", (0.0, 0.0))])
def test_rows_say_how_uniform_the_knots_are(knots, flags):
    n, end = 2000, 5.81
    x = {"linspace": np.linspace(0.0, end, n), "multiples": np.arange(n) * 2.9e-3,
         "summed": np.concatenate([[0.0], np.cumsum(np.full(n - 1, end / (n - 1)))]),
         "stretched": np.linspace(0.0, end, n), "uneven": np.linspace(0.0, 1.0, n) ** 1.05 * end}[knots]
    if knots == "stretched":
        t = x / end
        x = x + 9e-10 * t * (1.0 - t) * end
    spec = SpecFunction(("spline", x, np.ones((4, n - 1))))
    P = EAMPotential({"A": spec}, {"A": spec}, {("A", "A"): spec}, r_cut=5.0, species=["A"]).function_table()["P"]
    off = np.abs(x - (x[0] + np.arange(n) * (1.0 / P[0, 2]))).max() if P[0, 0] else np.inf
    assert P[0, 3] == (1.0 if off <= 4 * np.spacing(x.max()) else 0.0)
    if flags is not None:
        assert tuple(P[0, [0, 3]]) == flags
    assert (P[:, 4:] == 0.0).all()


@pytest.mark.gpu
@pytest.mark.parametrize("species", [["Ni"], ["Cu", "Ni"]])
def test_nearly_uniform_knots_match_the_oracle(cuda_device, species):
    pot = _stretched(_tables(species, n=1500), 9e-10)
    lat, pos, _ = cubic(FCC, 3.65, 5, ["X"] * 4, rattle=0.06, seed=2)
    ids = np.random.default_rng(4).integers(0, len(species), len(pos)).astype(np.int32)
    types = [species[k] for k in ids]
    e0, f0, _ = _oracle(pot, lat, pos, types)
    batch = ak.Batch.single(lat, pos, ids, device=cuda_device)
    dl = ak.DeviceNeighbourList(pot.r_cut + 0.2).build(batch)
    assert dl.n_slots >= 2 * pot.function_table()["X"].shape[0]   # long enough for packed tables
    r = pot.evaluate(batch, dl, precision="fp64")
    pot.status()
    top = max(1.0, np.abs(f0).max())
    assert abs(float(r.energy[0]) - e0) / len(pos) < 1e-11
    assert np.abs(r.forces.cpu().numpy() - f0).max() < 1e-10 * top
