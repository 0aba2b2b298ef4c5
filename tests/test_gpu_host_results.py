"""Host results of force calls stay the caller's: a later call, of the same
size or another, leaves arrays that are still held as they were; and the
batch's own copy of forces to the host gives the same values."""
import gc

import numpy as np
import pytest

from conftest import DIAMOND, cubic

pytestmark = pytest.mark.gpu

ak = pytest.importorskip("akitsushima_b200")


def test_results_are_not_overwritten(cuda_device):
    pot = ak.TersoffPotential(ak.TERSOFF_SI_1988, species=["Si"])
    held = []
    for k in range(6):
        lat, pos, _ = cubic(DIAMOND, 5.431, 2 + k % 2, ["Si"] * 8, rattle=0.05, seed=k)
        nl = ak.NeighbourList(pot.r_cut, skin_width=0.3)
        nl.build(lat, pos)
        e, f, s = pot.compute(lat, pos, np.zeros(len(pos), np.int32), nl)
        held.append((e, f, s, f.copy(), s.copy()))
        if k == 3:
            del held[1]                     # its block may be taken again
            gc.collect()
    for e, f, s, f0, s0 in held:
        np.testing.assert_array_equal(f, f0)
        np.testing.assert_array_equal(s, s0)
        assert f.flags.writeable and f.flags.c_contiguous and f.dtype == np.float64


def test_forces_to_host(cuda_device):
    pot = ak.TersoffPotential(ak.TERSOFF_SI_1988, species=["Si"])
    lat, pos, _ = cubic(DIAMOND, 5.431, 3, ["Si"] * 8, rattle=0.05, seed=1)
    batch = ak.Batch.single(lat, pos, np.zeros(len(pos), np.int32), device=cuda_device)
    r = pot.evaluate(batch, ak.DeviceNeighbourList(pot.r_cut + 0.3).build(batch))
    f = batch.forces_to_host(r.forces)
    np.testing.assert_array_equal(f, r.forces.cpu().numpy())
    assert f.shape == (len(pos), 3)
