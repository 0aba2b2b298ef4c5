"""The kick kernels at the edges of their blocks, through the C ABI: one
structure (128 atoms a block) and batches (1024 atoms a block, a block column
per structure) of sizes around both, against numpy: the half kick, the whole
kick and drift of the fused launch, and the kinetic energies.

Tolerances: a component is two or three rounded operations, 4 eps of the
operands' sizes (1e-15 of the largest); a kinetic energy is a sum of up to
3 N positive terms, N eps relative (1e-12).  The fused launch's thermo row has
the bits of the separate one.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ak = pytest.importorskip("akitsushima_b200")
from akitsushima_b200 import _lib  # noqa: E402

SIZES = [(1,), (127,), (128,), (129,), (1025,), (5000,), (1, 129, 1024), (1025, 3, 1023, 2049)]


@pytest.mark.parametrize("sizes", SIZES)
def test_kicks_match_numpy(cuda_device, sizes):
    L = _lib.lib()
    dev = cuda_device
    rng = np.random.default_rng(sum(sizes))
    n, ns, dt = sum(sizes), len(sizes), 0.7
    box = 40.0
    pos = rng.uniform(5.0, box - 5.0, (n, 3))
    batch = ak.Batch([np.eye(3) * box] * ns, np.split(pos, np.cumsum(sizes)[:-1]),
                     [np.zeros(k, np.int32) for k in sizes], device=dev)
    vel, frc, im = rng.normal(size=(n, 3)) * 0.01, rng.normal(size=(n, 3)), rng.uniform(0.2, 2.0, n) * 1e-3
    f64 = lambda x: torch.as_tensor(x, dtype=torch.float64, device=dev)  # noqa: E731
    v, F, w, E = f64(vel).clone(), f64(frc), f64(im), f64(rng.normal(size=ns))
    partial = torch.empty(ns * int(L.mbf_md_partial_count(n)), dtype=torch.float64, device=dev)
    thermo = torch.zeros((3, ns, 2), dtype=torch.float64, device=dev)
    words = torch.zeros(8, dtype=torch.int32, device=dev)
    word = lambda k: words.data_ptr() + 4 * k  # noqa: E731
    st = torch.cuda.current_stream(dev).cuda_stream
    sysd = batch.mbf_system()
    _lib.check(L.mbf_md_kick(sysd, _lib.ptr(v), _lib.ptr(F), _lib.ptr(w), dt, _lib.ptr(E), _lib.ptr(partial),
                             _lib.ptr(thermo), 3, word(0), word(6), st), "mbf_md_kick")
    half = vel + 0.5 * dt * im[:, None] * frc
    np.testing.assert_allclose(v.cpu().numpy(), half, rtol=0, atol=1e-15 * np.abs(half).max())
    ekin = [0.5 * np.sum((half[a:b] ** 2).sum(1) / im[a:b])
            for a, b in zip(np.cumsum((0,) + sizes), np.cumsum(sizes))]
    got = thermo[0].cpu().numpy()
    np.testing.assert_array_equal(got[:, 0], E.cpu().numpy())
    np.testing.assert_allclose(got[:, 1], ekin, rtol=1e-12)

    # the fused launch from the same start: the same thermo row, then the drift
    v.copy_(f64(vel))
    ref = batch.pos.clone()
    dmax = torch.zeros(ns, dtype=torch.float64, device=dev)
    log = torch.zeros((3, ns), dtype=torch.float64, device=dev)
    _lib.check(L.mbf_md_kick_kick_drift_check(
        sysd, _lib.ptr(batch.pos), _lib.ptr(v), _lib.ptr(F), _lib.ptr(w), dt, _lib.ptr(E), _lib.ptr(partial),
        _lib.ptr(thermo), 3, word(0), _lib.ptr(ref), 4.0, 3.7, _lib.ptr(dmax), _lib.ptr(log), 3, word(1), word(4), 0,
        word(5), st), "mbf_md_kick_kick_drift_check")
    full = half + 0.5 * dt * im[:, None] * frc
    np.testing.assert_allclose(v.cpu().numpy(), full, rtol=0, atol=1e-15 * np.abs(full).max())
    moved = pos + dt * full
    np.testing.assert_allclose(batch.pos.cpu().numpy(), moved, rtol=0, atol=1e-15 * box * 8)
    assert torch.equal(thermo[1], thermo[0])
    w_ = words.cpu().numpy()
    far = [np.sqrt((((dt * full) ** 2).sum(1))[a:b].max()) for a, b in zip(np.cumsum((0,) + sizes), np.cumsum(sizes))]
    np.testing.assert_allclose(log[0].cpu().numpy(), far, rtol=0, atol=1e-15 * box * 8)
    assert w_[0] == 2 and w_[1] == 1 and w_[4] == int(max(far) * 2 >= 0.3) and w_[5] == 0 and w_[6] == 0
