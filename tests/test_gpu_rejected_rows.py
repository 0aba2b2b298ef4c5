"""Rows that the three-body evaluations reject (a species outside the tables,
row bounds outside the slots): the status says so, and nothing that an earlier
evaluation, or nobody, left in the workspace reaches the forces through the
row's live mask."""
import numpy as np
import pytest
import torch

from conftest import DIAMOND, SW_SI, cubic

pytestmark = pytest.mark.gpu

ak = pytest.importorskip("akitsushima_b200")
from akitsushima_b200 import _lib  # noqa: E402


@pytest.mark.parametrize("radius", [4.1, 5.9])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", ["sw", "tersoff"])
def test_rejected_rows_add_nothing(cuda_device, name, precision, radius):
    lat, pos, _ = cubic(DIAMOND, 5.431, 3, ["Si"] * 8, rattle=0.05, seed=6)
    pot = ak.StillingerWeberPotential(SW_SI, species=["Si"]) if name == "sw" else \
        ak.TersoffPotential(ak.TERSOFF_SI_1988, species=["Si"])
    n = len(pos)
    for what in ("species", "begin", "end"):
        batch = ak.Batch.single(lat, pos, np.zeros(n, np.int32), device=cuda_device)
        dl = ak.DeviceNeighbourList(radius).build(batch)
        ws = torch.empty(int(_lib.lib().mbf_eval_workspace_bytes(n, dl.n_slots, batch.n_chunks)), dtype=torch.uint8,
                         device=cuda_device)
        ws.fill_(255)                       # NaN in every double, every live bit set
        if what == "species":
            batch.types[7] = 3
        elif what == "begin":
            dl.row_off[7] = -(1 << 30)      # rows 6 and 7
        else:
            dl.row_off[n] = 1 << 30         # the last row
        r = pot.evaluate(batch, dl, precision=precision, ws=ws)
        with pytest.raises(RuntimeError, match="device check failed"):
            pot.status()
        rejected = {"species": [7], "begin": [6, 7], "end": [n - 1]}[what]
        f = r.forces.cpu().numpy()
        np.testing.assert_array_equal(f[rejected], 0.0)
        if what == "species":               # its neighbours do not read its slots either
            assert np.isfinite(f).all()
