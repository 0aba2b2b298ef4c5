"""The Tersoff adjoint's angular derivatives on isolated trimers, one centre
with two legs that do not see each other, against the closed form in long
double: no cancellation may cost digits where h - cos is small beside d.

With E = sum over the two bonds of 1/2 fc (fR + b fA), b = (1 + (beta z)^n)^
(-1 / 2n) and z_j = gamma fc(r_k) g, dE/dp = 1/2 fc fA db/dz dz/dp.  Tolerance:
cos carries a few 1e-16, h - cos down to 0.05 so a part in 1e-14 at most, its
square twice that; 5e-14 relative.  2 d / q^2 - 2 / d^3 taken as a difference
is off by 1e-13 to 1e-11 here.
"""
import numpy as np
import pytest
import torch

from conftest import TERSOFF_SI

pytestmark = pytest.mark.gpu

ak = pytest.importorskip("akitsushima_b200")
from akitsushima_b200 import fit  # noqa: E402

ld = np.longdouble


@pytest.mark.parametrize("cos", [-0.99, -0.8, -0.65, -0.55, -0.45, -0.3, -0.1])
def test_trimer_angular_derivatives(cuda_device, cos):
    p = dict(TERSOFF_SI, m=3.0, gamma=1.0)
    ra, rb = 2.25, 2.4                                    # inside R - D = 2.7: fc = 1
    assert ra * ra + rb * rb - 2 * ra * rb * cos > 3.0 ** 2   # the legs' ends are out of reach
    pos = np.array([[0.0, 0.0, 0.0], [ra, 0.0, 0.0], [rb * cos, rb * np.sqrt(1 - cos * cos), 0.0]]) + 20.0
    tb = torch.tensor([[1.0, p["A"], p["B"], p["lambda1"], p["lambda2"], p["R"], p["D"], p["beta"], p["n"], 0.0]],
                      dtype=torch.float64, device=cuda_device)
    tri = torch.tensor([[1.0, p["c"], p["d"], p["h"], 0.0, 3.0, 1.0, 0.0]], dtype=torch.float64, device=cuda_device)
    ev = fit._TableEval(ak.Batch.single(np.eye(3) * 40.0, pos, np.zeros(3, np.int32), device=cuda_device), 0.3)
    ev.evaluate(tb, tri, 3.0)
    gE = torch.ones(1, dtype=torch.float64, device=cuda_device)
    d_tri = ev.adjoint(tb, tri, gE, None, None, r_cut=3.0)[1].cpu().numpy()[0]
    d = (pos[1:] - pos[0]).astype(ld)
    r = np.sqrt((d * d).sum(1))
    hc = ld(p["h"]) - (d[0] * d[1]).sum() / (r[0] * r[1])
    c, dd, beta, n = (ld(p[k]) for k in ("c", "d", "beta", "n"))
    q = dd * dd + hc * hc
    z = 1 + c * c / (dd * dd) - c * c / q
    u = (beta * z) ** n
    dbdz = -u * (1 + u) ** (-1 / (2 * n) - 1) / (2 * z)
    fA = -ld(p["B"]) * np.exp(-ld(p["lambda2"]) * r)
    w = (fA * dbdz / 2).sum()
    want = {1: w * 2 * c * (1 / (dd * dd) - 1 / q), 2: w * c * c * (2 * dd / q ** 2 - 2 / dd ** 3),
            3: w * 2 * c * c * hc / q ** 2}
    for col, v in want.items():
        assert abs(d_tri[col] - float(v)) <= 5e-14 * abs(float(v)), col
