"""The narrow transport (a disk alone) against the wide one (the same disk beside
one large enough to fill the chip): the same bits, at ring counts that leave a
band with fewer rings than a half-band, and at sector counts around one and two
narrow segments and their windows."""
import numpy as np
import pytest

from cudaprotoplanetarydisksfloat_b200 import Batch, Disk, noise
from tests.helpers import SEED, small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["iso", "adi"])
@pytest.mark.parametrize("nrad,nsec", [(8, 64), (5, 112), (12, 120), (13, 124), (9, 240), (20, 244), (17, 364)])
def test_narrow_equals_wide(gpu, kind, nrad, nsec):
    P, L, _ = small(kind, nrad, nsec)
    Q, M, _ = small(kind, 320, 2000, DT="0.001")
    d = Disk(P, L)
    dens = noise.perturb_density(d.fields()["dens"].reshape(-1), nrad, nsec, SEED)
    d.init_state(dens=dens)
    b = Batch([P, Q], [L, M])
    b.init_state(0, dens=dens)
    d.advance(1)
    b.advance(1)
    assert d.scalars()["nsub_last_dt"] == b.scalars(0)["nsub_last_dt"]
    x, y = d.fields(), b.fields(0)
    for k in x:
        assert np.array_equal(x[k], y[k]), k
