"""The Tersoff adjoint's bond lists at their edges, against central
differences of the evaluation: one and three species, absent records, lambda3
with the first, second and third power, each upstream gradient alone, atoms
without neighbours (fewer slots than atoms) and more slots than one tile of
the partition.

Tolerance as tests/test_gpu_fit.py: 1e-6 relative, or 1e-6 of a thousandth of
the largest entry; steps of 1e-5 relative, summed result by result.
"""
import numpy as np
import pytest
import torch

from conftest import DIAMOND, cubic, strained
from test_gpu_tersoff_center import _records

pytestmark = pytest.mark.gpu

ak = pytest.importorskip("akitsushima_b200")
from akitsushima_b200 import fit  # noqa: E402

CASES = {
    # name: (species, record options, lattice constant, cells, upstream gradients)
    "one": (1, {}, 5.3, 3, "EFW"),
    "three": (3, dict(drop=4), 5.1, 3, "EFW"),
    "m1": (2, dict(lam=0.4, m=1.0), 5.1, 2, "EFW"),
    "m2": (2, dict(lam=0.5, m=2.0), 5.1, 2, "EFW"),
    "m3": (2, dict(lam=1.2, m=3.0), 5.1, 2, "EFW"),
    "forces_only": (2, {}, 5.1, 2, "F"),
    "energy_and_virial": (2, {}, 5.1, 2, "EW"),
    "isolated": (2, {}, 9.0, 2, "EFW"),
}


@pytest.mark.parametrize("name", list(CASES))
def test_adjoint_lists_match_central_differences(cuda_device, name):
    ns, opts, a, cells, grads = CASES[name]
    sp, rec = _records(ns, 3, **opts)
    structs = []
    for k in range(2):
        L, P, _ = cubic(DIAMOND, a, cells, ["x"] * 8, rattle=0.08, seed=20 + k)
        L, P = strained(L, P, 0.01, 30 + k)
        P = P[:len(P) - 3 * k - 1]
        if name == "isolated" and k == 0:
            P[1] = P[0] + [2.3, 0.1, 0.0]       # one bonded pair in a gas
        structs.append((L, P, np.random.default_rng(40 + k).integers(0, ns, len(P)).astype(np.int32)))
    batch = ak.Batch([s[0] for s in structs], [s[1] for s in structs], [s[2] for s in structs], device=cuda_device)
    ev = fit._TableEval(batch, 0.3)
    tabs = [t.to(cuda_device) for t in fit.tables_from_records(rec, sp, "cpu")]
    E, F, W = ev.evaluate(*tabs)
    if name == "isolated":
        assert ev.dlist.n_slots < batch.n_atoms
    rng = np.random.default_rng(5)
    g = {k: torch.as_tensor(rng.normal(size=v.shape), device=cuda_device) for k, v in zip("EFW", (E, F, W))}
    up = [g[k] if k in grads else None for k in "EFW"]
    rc = fit.table_cutoff(tabs[0])
    got = ev.adjoint(*tabs, *up, r_cut=rc)
    again = ev.adjoint(*tabs, *up, r_cut=rc)
    assert all(torch.equal(u, v) for u, v in zip(got, again))
    top = max(float(t.abs().max()) for t in got)
    cols = {0: range(1, 9), 1: (1, 2, 3, 4, 6)}
    bad = []
    for which in (0, 1):
        for row in range(tabs[which].shape[0]):
            for col in range(tabs[which].shape[1]):
                d = float(got[which][row, col])
                if col not in cols[which] or float(tabs[which][row, 0]) == 0.0:
                    assert d == 0.0
                    continue
                v = float(tabs[which][row, col])
                if which == 1 and col == 4 and v == 0.0 and opts.get("m", 3.0) != 1.0:
                    continue                    # (lambda3 u)^3 has no slope at 0
                h = 1e-5 * abs(v) if v != 0.0 else 1e-5
                res = []
                for s in (h, -h):
                    t = [x.clone() for x in tabs]
                    t[which][row, col] += s
                    res.append([x.clone() for x in ev.evaluate(*t, r_cut=rc)])
                fd = sum(float((u * (p - m)).sum()) for u, p, m in zip(up, *res) if u is not None) / (2 * h)
                if abs(d - fd) > 1e-6 * max(abs(fd), 1e-3 * top):
                    bad.append((which, row, col, d, fd))
    assert not bad, bad[:5]
