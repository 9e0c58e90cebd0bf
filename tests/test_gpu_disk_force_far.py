"""The disk force where the Hill cut's exponent -d^2 / rh^2 overflows: a body at
the origin or without mass has a cut radius of 1e-15, and the cells of a disk
in large length units lie thousands of units away.  The quotient is then -inf
and the cut 1, as in the oracle: every sum finite, and within the 1e-6 of the
sums' scale that the other disk-force tests allow (the same FP32 forces summed
in FP64).  The density has an m = 1 mode, so that the sums at the origin do not
cancel."""
import numpy as np
import pytest

from cudaprotoplanetarydisksfloat_b200 import Disk
from oracle.oracle import Oracle
from tests.helpers import rel_l2, small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x,y,m", [(0.0, 0.0, 1e-3), (0.0, 0.0, 0.0), (1500.0, 0.0, 0.0), (0.0, -5100.0, 0.0)])
def test_far_cells(gpu, x, y, m):
    nrad, nsec = 16, 64
    P, L, _ = small("iso", nrad, nsec, Rmin="500.0", Rmax="5000.0")
    d, o = Disk(P, L), Oracle(P, L)
    mode = 1.0 + 0.5 * np.cos(2 * np.pi * np.arange(nsec) / nsec)
    d.init_state(dens=(d.fields()["dens"] * mode).astype(np.float32).reshape(-1))
    o.set_fields(**{k: v for k, v in d.fields().items() if k in ("dens", "vrad", "vtheta", "energy")})
    a, b = d.disk_force(x, y, 20.0, m), o.disk_force(x, y, 20.0, m)
    assert np.isfinite(b).all()
    assert np.isfinite(a).all()
    assert rel_l2(a, b) <= 1e-6
