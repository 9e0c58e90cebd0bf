"""The element-wise self-gravity kernels on rings that are no whole 16-byte words
(NSEC not a multiple of 4) and at the edges of their blocks, against the FP64
oracle.  In the accurate mode the kernel table is FP64's, so what is left is
the FP32 transforms' rounding: 2^-24 times the log2 of the padded grid's size,
about 1.2e-6 of the transforms' scale.  That scale is g_r's for both fields: the
density is an axisymmetric profile with 1e-3 of noise, and g_phi, which only the
noise makes, is what is left of terms a thousand times larger.  A DT of the reference mode
(the edge rings' means enter its boundary) is held to the parity tests' bounds."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from tests.helpers import rel_l2
from tests.test_gpu_parity import _compare, _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrad,nsec", [(20, 66), (33, 67), (16, 64), (24, 253), (9, 1028)])
def test_accelerations_vs_fp64(gpu, nrad, nsec):
    P, L, d, o, dens = _pair("sg", nrad, nsec)
    d.set_precision(1)
    o64 = Oracle(P, L, "f64")
    o64.set_precision(1)
    g = d.fields()
    o64.set_fields(dens=g["dens"], vrad=g["vrad"], vtheta=g["vtheta"], energy=g["energy"])
    a, w = d.sg_accelerations(), o64.sg_accelerations()
    assert rel_l2(a[0], w[0]) <= 1.2e-6
    assert np.linalg.norm(a[1].astype(np.float64) - w[1]) <= 1.2e-6 * np.linalg.norm(w[0])


def test_odd_ring_parity(gpu):
    P, L, d, o, _ = _pair("sg", 32, 66)
    _compare(P, d, o, 2, planet_rtol=1e-5)
