"""Mass of a disk with rigid edges over many substeps.  What leaves a cell enters
its neighbour, so the mass changes by roundings alone: a cell is updated three
times a substep (radially, and by the two azimuthal sweeps), each to within 2^-24
of its value, and at the edges of the isothermal transport's bands of 8 rings the
two sides of an interface may differ by a rounding of what crosses it, which is
less than half a ring.  In the worst case, all of one sign: 3.5 * 2^-24 of the mass
a substep; the bound is 4.  Narrow and wide transport, ring counts with and without
a partial last band."""
import numpy as np
import pytest

from cudaprotoplanetarydisksfloat_b200 import Disk, grid_radii, noise
from tests.helpers import SEED, small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nrad,nsec,ndt", [
    ("iso", 64, 192, 20), ("iso", 61, 190, 20), ("iso", 512, 1000, 3), ("adi", 64, 192, 20)])
def test_mass_is_kept(gpu, kind, nrad, nsec, ndt):
    P, L, _ = small(kind, nrad, nsec)
    d = Disk(P, L)
    d.init_state(dens=noise.perturb_density(d.fields()["dens"].reshape(-1), nrad, nsec, SEED))
    R = np.array(grid_radii(P), np.float64)
    # the FP32 ring areas the kernels use
    surf = (np.pi * (R[1:] ** 2 - R[:-1] ** 2) / nsec).astype(np.float32).astype(np.float64)
    mass = lambda: float((d.fields()["dens"][:nrad].astype(np.float64) * surf[:, None]).sum())  # noqa: E731
    m0 = mass()
    for _ in range(ndt):
        d.advance_dt()
    n, drift = d.scalars()["nsub_total"], abs(mass() / m0 - 1.0)
    print("\n%s %dx%d: %d substeps, mass %.1e" % (kind, nrad, nsec, n, drift))
    assert n >= 50
    assert drift <= 4 * n * 2.0 ** -24
