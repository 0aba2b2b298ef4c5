"""Three-body evaluations, their site terms and the Tersoff adjoint in a
workspace that starts at an odd multiple of 8 bytes, of exactly the bytes
asked for: the bits of an aligned one."""
import numpy as np
import pytest
import torch

from conftest import DIAMOND, SW_SI, cubic

pytestmark = pytest.mark.gpu

ak = pytest.importorskip("akitsushima_b200")
from akitsushima_b200 import _lib, fit  # noqa: E402
from test_gpu_tersoff_center import _records  # noqa: E402


def _odd(nbytes, device):
    """nbytes at an address that is 8 modulo 16, with guard bytes behind."""
    whole = torch.full((nbytes + 64,), 255, dtype=torch.uint8, device=device)
    assert whole.data_ptr() % 16 == 0
    return whole[8:8 + nbytes], whole[8 + nbytes:]


@pytest.mark.parametrize("n_drop", [0, 3, 8])      # with and without slack behind the masks
@pytest.mark.parametrize("name", ["sw", "tersoff"])
def test_eval_in_an_odd_workspace(cuda_device, name, n_drop):
    lat, pos, _ = cubic(DIAMOND, 5.431, 4, ["Si"] * 8, rattle=0.08, seed=6)
    pos = pos[:len(pos) - n_drop]
    pot = ak.StillingerWeberPotential(SW_SI, species=["Si"]) if name == "sw" else \
        ak.TersoffPotential(ak.TERSOFF_SI_1988, species=["Si"])
    batch = ak.Batch.single(lat, pos, np.zeros(len(pos), np.int32), device=cuda_device)
    dl = ak.DeviceNeighbourList(pot.r_cut + 0.3).build(batch)
    ref = pot.evaluate(batch, dl)
    pot.status()
    ws, guard = _odd(int(_lib.lib().mbf_eval_workspace_bytes(len(pos), dl.n_slots, batch.n_chunks)), cuda_device)
    got = pot.evaluate(batch, dl, ws=ws)
    pot.status()
    for key in ("energy", "forces", "virial"):
        assert torch.equal(getattr(ref, key), getattr(got, key))
    assert bool((guard == 255).all())


@pytest.mark.parametrize("ns", [1, 3])
def test_tersoff_adjoint_in_an_odd_workspace(cuda_device, ns):
    sp, rec = _records(ns, 3)
    lat, pos, _ = cubic(DIAMOND, 5.2, 3, ["x"] * 8, rattle=0.08, seed=20)
    batch = ak.Batch.single(lat, pos, np.random.default_rng(1).integers(0, ns, len(pos)).astype(np.int32),
                            device=cuda_device)
    ev = fit._TableEval(batch, 0.3)
    tabs = [t.to(cuda_device) for t in fit.tables_from_records(rec, sp, "cpu")]
    up = ev.evaluate(*tabs)
    rc = fit.table_cutoff(tabs[0])
    ref = ev.adjoint(*tabs, *up, r_cut=rc)
    ev._adj_ws, guard = _odd(int(_lib.lib().mbf_tersoff_adjoint_workspace_bytes(ev.dlist.n_slots, ns)), cuda_device)
    got = ev.adjoint(*tabs, *up, r_cut=rc)
    for a, b in zip(ref, got):
        assert torch.equal(a, b)
    assert bool((guard == 255).all())
