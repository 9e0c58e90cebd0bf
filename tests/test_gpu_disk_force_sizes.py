"""The disk-force sums where their blocks and sides can go wrong, against the
oracle's: fewer cells than a block, runs that end inside a ring, a body inside
the first ring (every cell outer), outside the last (every cell inner) and
between two, repeated calls (the ticket).  The same FP32 forces summed in FP64:
the bound is 1e-6 of the sums' scale, as in the parity test of this call."""
import numpy as np
import pytest

from tests.helpers import rel_l2
from tests.test_gpu_parity import _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrad,nsec", [(4, 32), (16, 64), (31, 67), (33, 130), (300, 130)])
def test_force_sides_and_runs(gpu, nrad, nsec):
    P, L, d, o, _ = _pair("iso", nrad, nsec)
    for x, y, rs, m in [(0.1, 0.0, 0.02, 1e-4), (3.0, 1.0, 0.1, 1e-3), (1.0, 0.2, 0.03, 1e-3), (0.0, 0.8, 0.05, 0.0)]:
        for _ in range(2):
            a = d.disk_force(x, y, rs, m)
        b = o.disk_force(x, y, rs, m)
        assert rel_l2(a, b) <= 1e-6
        assert np.array_equal(np.abs(a) > 0, np.abs(b) > 0)
