"""The kick kernels on both sides of the line between an atom a thread and four
(65,536 atoms of one structure), and batches, whose partial sums fit the
counts asked for: against numpy, tolerances as test_gpu_md_kick_blocks."""
import pytest

from test_gpu_md_kick_blocks import test_kicks_match_numpy as _kicks
from akitsushima_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(65535,), (65536,), (65537,), (131073,), (70000, 5)])
def test_kicks_across_the_line(cuda_device, sizes):
    _kicks(cuda_device, sizes)


def test_partial_counts():
    """One partial per 128 atoms up to the line, one per 1024 beyond; never
    fewer than a batch of as many atoms needs."""
    L = _lib.lib()
    for n, want in ((0, 1), (1, 1), (129, 2), (65536, 512), (65537, 65), (1 << 20, 1024)):
        assert L.mbf_md_partial_count(n) == want
        assert want >= -(-n // 1024)
