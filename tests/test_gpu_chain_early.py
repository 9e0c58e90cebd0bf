"""Kernels of one disk that begin before the kernel ahead of them has ended: the
CFL kernel forms the disk force while the ring means are summed, the potential
kernel the first bodies' terms while the substep's scalars are finished, the
transport its first items' radial half while the shifts are summed.  Beside a
second disk the same kernels wait at their start: the same operations in the
same order, so the same bits.  Up to four bodies' terms are formed early (0 to 6
planets beside the star's own term), the potential only where each block has a
tile at most (the last two grids have more); an NSEC of odd quads takes the
wait at the start."""
import numpy as np
import pytest

from cudaprotoplanetarydisksfloat_b200 import Batch, Disk, configs, noise
from cudaprotoplanetarydisksfloat_b200.disk import planets_dict
from tests.helpers import SEED, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nrad,nsec,npl", [
    ("iso", 8, 64, 0), ("iso", 33, 96, 1), ("adi", 33, 96, 3), ("adi", 40, 128, 4), ("adi", 40, 128, 5),
    ("iso", 24, 260, 6), ("iso", 31, 101, 2), ("iso", 700, 2048, 2), ("adi", 700, 2048, 5)])
def test_alone_equals_beside_another(gpu, kind, nrad, nsec, npl):
    p, _ = configs.small(kind, nrad, nsec)
    p = dict(p, DT="0.002" if nrad > 100 else "0.1", ForcedCircular="NO")
    pl = [("P%d" % k, 0.7 + 0.3 * k, 1e-4 * (k + 1), "YES" if k < 5 else "NO", "YES") for k in range(npl)]
    P, L = make(p, pl, kind)[:2]
    d = Disk(P, L)
    dens = noise.perturb_density(d.fields()["dens"].reshape(-1), nrad, nsec, SEED)
    d.init_state(dens=dens)
    b = Batch([P, P], [L, L])
    for k in range(2):
        b.init_state(k, dens=dens)
    d.advance(2)
    b.advance(2)
    assert d.scalars()["nsub_total"] == b.scalars(1)["nsub_total"]
    x, y = d.fields(), b.fields(1)
    for k in x:
        assert np.array_equal(x[k], y[k]), k
    u, v = planets_dict(d.planets()), planets_dict(b.planets(1))
    for k in u:
        assert np.array_equal(u[k], v[k]), k
