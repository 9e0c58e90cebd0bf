"""A disk with both the damping zones and an open or non-reflecting edge (the
.par file names one boundary; the parameter block of the C interface can set
two).  The damping of a disk's rings comes first, by many blocks, and the edge
rings after all of them: an open edge then leaves ring 0 as the copy of the
damped ring 1, a non-reflecting one leaves ring 0 with the mean of the initial
profile, whatever the blocks' order."""
import numpy as np
import pytest

from cudaprotoplanetarydisksfloat_b200 import Disk, noise
from tests.helpers import SEED, small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["iso", "adi"])
@pytest.mark.parametrize("nrad,nsec", [(40, 130), (200, 516)])
def test_open_edge_follows_the_damping(gpu, kind, nrad, nsec):
    P, L, _ = small(kind, nrad, nsec, InnerBoundary="EVANESCENT")
    P.OpenInner = 1
    d = Disk(P, L)
    d.init_state(dens=noise.perturb_density(d.fields()["dens"].reshape(-1), nrad, nsec, SEED))
    for _ in range(3):
        d.advance_dt()
        f = d.fields()
        assert np.array_equal(f["dens"][0], f["dens"][1])
        if kind == "adi":
            assert np.array_equal(f["energy"][0], f["energy"][1])


@pytest.mark.parametrize("kind", ["iso", "adi"])
def test_non_reflecting_edge_follows_the_damping(gpu, kind):
    nrad, nsec = 200, 516
    P, L, _ = small(kind, nrad, nsec, InnerBoundary="EVANESCENT")
    P.NonReflecting = 1
    d = Disk(P, L)
    profile = d.fields()["dens"].astype(np.float64).mean(axis=1)
    dens = noise.perturb_density(d.fields()["dens"].reshape(-1), nrad, nsec, SEED)
    d.init_state(dens=dens)
    e = Disk(P, L)
    e.init_state(dens=dens)
    for _ in range(2):
        d.advance_dt()
        e.advance_dt()
    f, g = d.fields(), e.fields()
    # the ring is shifted to the profile's mean: an FP32 sum of 516 values and one addition each
    assert abs(f["dens"][0].astype(np.float64).mean() / profile[0] - 1.0) <= 516 * 2.0 ** -24
    for k in f:
        assert np.array_equal(f[k], g[k]), k
