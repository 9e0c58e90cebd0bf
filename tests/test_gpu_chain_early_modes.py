"""The early starts of a disk alone (test_gpu_chain_early.py) in the forms that
change the kernels around them: boundary calls between the kernels, the accurate
mode's kernels, a corotating frame (the planets before the source terms), cooling
and self-gravity beside the chain.  Beside a second disk the same kernels wait at
their start: the same bits."""
import numpy as np
import pytest

from cudaprotoplanetarydisksfloat_b200 import Batch, Disk, noise
from cudaprotoplanetarydisksfloat_b200.disk import planets_dict
from tests.helpers import SEED, small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nrad,nsec,accurate,over", [
    ("iso", 33, 132, False, {"InnerBoundary": "NONREFLECTING"}),
    ("iso", 40, 260, False, {"InnerBoundary": "EVANESCENT", "Frame": "COROTATING"}),
    ("iso", 24, 200, False, {"InnerBoundary": "OPEN"}),
    ("adi", 33, 132, False, {"InnerBoundary": "NONREFLECTING"}),
    ("adi", 40, 128, False, {"InnerBoundary": "EVANESCENT"}),
    ("adi", 40, 128, False, {"Cooling": "YES", "Frame": "COROTATING"}),
    ("iso", 33, 96, True, {}),
    ("iso", 8, 48, True, {}),
    ("iso", 31, 101, True, {}),
    ("adi", 33, 96, True, {}),
    ("iso", 33, 132, True, {"InnerBoundary": "EVANESCENT"}),
    ("sg", 32, 96, False, {}),
    ("sg", 32, 96, True, {})])
def test_alone_equals_beside_another(gpu, kind, nrad, nsec, accurate, over):
    P, L, _ = small(kind, nrad, nsec, **over)
    d, b = Disk(P, L), Batch([P, P], [L, L])
    if accurate:
        d.set_precision(1)
        b.set_precision(1)
    dens = noise.perturb_density(d.fields()["dens"].reshape(-1), nrad, nsec, SEED)
    d.init_state(dens=dens)
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
