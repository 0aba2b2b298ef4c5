"""The Tersoff adjoint of tables with a sharp cutoff (D = 0): the cutoff
function is 1 up to R and 0 beyond, so without a neighbour at R itself its
derivatives in R and D vanish and every other entry is that of a cutoff of
vanishing width (1e-9 A, whose window holds no neighbour)."""
import numpy as np
import pytest
import torch

from conftest import DIAMOND, cubic, strained
from test_gpu_tersoff_center import _records

pytestmark = pytest.mark.gpu

ak = pytest.importorskip("akitsushima_b200")
from akitsushima_b200 import fit  # noqa: E402


@pytest.mark.parametrize("ns,opts", [(1, {}), (2, dict(lam=1.2, m=3.0)), (3, dict(drop=4))])
def test_sharp_cutoff(cuda_device, ns, opts):
    sp, rec = _records(ns, 3, **opts)
    L, P, _ = cubic(DIAMOND, 5.2, 3, ["x"] * 8, rattle=0.08, seed=20)
    L, P = strained(L, P, 0.01, 30)
    ids = np.random.default_rng(40).integers(0, ns, len(P)).astype(np.int32)
    ev = fit._TableEval(ak.Batch.single(L, P, ids, device=cuda_device), 0.3)
    tabs = [t.to(cuda_device) for t in fit.tables_from_records(rec, sp, "cpu")]
    grads = {}
    for D in (0.0, 1e-9):
        tb = tabs[0].clone()
        tb[:, 6] = D
        rc = float(tb[:, 5].max()) + 1e-6
        E, F, W = ev.evaluate(tb, tabs[1], rc)
        rng = np.random.default_rng(5)
        up = [torch.as_tensor(rng.normal(size=v.shape), device=cuda_device) for v in (E, F, W)]
        grads[D] = [t.cpu().numpy() for t in ev.adjoint(tb, tabs[1], *up, r_cut=rc)]
        np.testing.assert_array_equal(grads[D][0][:, 5:7], 0.0)
    for sharp, thin in zip(grads[0.0], grads[1e-9]):
        assert np.abs(thin).max() > 0.0
        np.testing.assert_array_equal(sharp, thin)
