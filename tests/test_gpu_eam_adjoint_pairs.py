"""The Zhou EAM adjoint's species-pair lists at their edges, against central
differences of the generic evaluation: one species (no cross list), five (two
packed count words), density rows that are not those of the pair rows, each
upstream gradient alone, and atom counts that fill no block.

Tolerance as tests/test_gpu_fit_eam.py: 1e-6 relative, or 1e-6 of a thousandth
of the largest entry.  The differences take steps of 1e-5 relative and are
summed result by result: at 1e-6 the rounding of an energy of 900 eV alone is
2e-7 of an entry of unit size, and at 1e-4 atoms cross the embedding's branch
points, where rows perturbed one by one are not continuous.
"""
import numpy as np
import pytest
import torch

from conftest import FCC, cubic, strained
from test_gpu_fit_eam import COLS

pytestmark = pytest.mark.gpu

ak = pytest.importorskip("akitsushima_b200")
from akitsushima_b200 import fit  # noqa: E402
from akitsushima_b200.published_parameters import ZHOU_2004  # noqa: E402

CASES = {
    # name: (species, rows perturbed one by one, upstream gradients, rows checked at most)
    "one": (["Ni"], 0.0, "EFW", 99),
    "rows_differ": (["Cu", "Ni"], 0.01, "EFW", 99),
    "forces_only": (["Cu", "Ni"], 0.0, "F", 99),
    "energy_and_virial": (["Cu", "Ni"], 0.0, "EW", 99),
    "five": (["Cu", "Ni", "Ag", "Pd", "Au"], 0.005, "EFW", 6),
}


@pytest.mark.parametrize("name", list(CASES))
def test_adjoint_lists_match_central_differences(cuda_device, name):
    sp, amp, grads, n_rows = CASES[name]
    ps = fit.ZhouEAMParameterSet({s: dict(ZHOU_2004[s]) for s in sp}, sp)
    skel = ps.potential().function_table()
    structs = []
    for k in range(2):
        L, P, _ = cubic(FCC, 3.75, 4, ["x"] * 4, rattle=0.07, seed=20 + k)
        L, P = strained(L, P, 0.01, 30 + k)
        P = P[:len(P) - 3 * k - 1]
        structs.append((L, P, np.random.default_rng(40 + k).integers(0, len(sp), len(P)).astype(np.int32)))
    batch = ak.Batch([s[0] for s in structs], [s[1] for s in structs], [s[2] for s in structs], device=cuda_device)
    ev = fit._EamTableEval(batch, 0.2, skel, ps.r_cut)
    ev.fused = 0   # the generic evaluation reads each row as the adjoint differentiates it
    P = ps.table_torch(torch.as_tensor(ps.x0))
    if amp:
        u = torch.as_tensor(np.random.default_rng(50).uniform(1 - amp, 1 + amp, P.shape))
        u[:, 40:42] = 1.0                       # one switch
        P = P * u
    P = P.contiguous().to(cuda_device)
    E, F, W = ev.evaluate(P)
    rng = np.random.default_rng(5)
    g = {k: torch.as_tensor(rng.normal(size=v.shape), device=cuda_device) for k, v in zip("EFW", (E, F, W))}
    up = [g[k] if k in grads else None for k in "EFW"]
    d_P = ev.adjoint(P, *up)
    assert torch.equal(d_P, ev.adjoint(P, *up))

    def slope(row, col, h):
        Pp, Pm = P.clone(), P.clone()
        Pp[row, col] += h
        Pm[row, col] -= h
        plus = [t.clone() for t in ev.evaluate(Pp)]
        return sum(float((u * (v - w)).sum()) for u, v, w in zip(up, plus, ev.evaluate(Pm)) if u is not None) / (2 * h)

    codes = skel["codes"]
    checks = []
    rows = range(P.shape[0]) if P.shape[0] <= n_rows else rng.choice(P.shape[0], n_rows, replace=False)
    for row in rows:
        for col in range(P.shape[1]):
            if col not in COLS[int(codes[row])]:
                assert float(d_P[row, col]) == 0.0
                continue
            v = float(P[row, col])
            checks.append((int(row), col, float(d_P[row, col]), slope(row, col, 1e-5 * abs(v) if v != 0.0 else 1e-5)))
    scale = float(d_P.abs().max())
    bad = [c for c in checks if abs(c[2] - c[3]) > 1e-6 * max(abs(c[3]), 1e-3 * scale)]
    assert not bad, bad[:5]


def test_host_rows_give_the_same_evaluation(cuda_device):
    """The fit's evaluation with its constants as kernel arguments (one and two
    species) against the shared-memory path."""
    for sp in (["Ni"], ["Al", "Ni"]):
        ps = fit.ZhouEAMParameterSet({s: dict(ZHOU_2004[s]) for s in sp}, sp)
        L, P, _ = cubic(FCC, 3.6, 5, ["x"] * 4, rattle=0.07, seed=3)
        ids = np.random.default_rng(4).integers(0, len(sp), len(P)).astype(np.int32)
        ev = fit._EamTableEval(ak.Batch.single(L, P, ids, device=cuda_device), 0.2,
                               ps.potential().function_table(), ps.r_cut)
        rows = ps.tables_np(ps.x0)[0]
        dev = torch.from_numpy(rows).to(cuda_device)
        a = [t.clone() for t in ev.evaluate(dev)]
        b = ev.evaluate(dev, np.ascontiguousarray(rows))
        for u, v in zip(a, b):
            assert float((u - v).abs().max()) <= 1e-12 * max(1.0, float(u.abs().max()))
