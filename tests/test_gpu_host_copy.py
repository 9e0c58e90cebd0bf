"""Field downloads: the driver's own path and the page-locked ring give what was
uploaded, bit for bit, at sizes around the thresholds and pieces that end
inside a page, into fresh and into touched buffers, from one thread and from
two at once (one of them then takes the plain path)."""
import ctypes as C
import threading

import numpy as np
import pytest

from cudaprotoplanetarydisksfloat_b200 import Disk
from cudaprotoplanetarydisksfloat_b200._abi import lib
from tests.helpers import small

pytestmark = pytest.mark.gpu

FIELDS = ("dens", "vrad", "vtheta", "energy")


def _disk(nrad, nsec, seed):
    P, L, _ = small("iso", nrad, nsec)
    d = Disk(P, L)
    rng = np.random.default_rng(seed)
    f = {k: rng.random((nrad + 1, nsec), dtype=np.float32) for k in FIELDS}
    d.upload(**f)
    return d, f


# 4 fields: 1.9 MB, 2.1 MB, an odd 9 MB, 25 MB (past the touched buffers' threshold)
@pytest.mark.parametrize("nrad,nsec", [(230, 513), (255, 513), (749, 751), (1200, 1301)])
def test_download_is_exact(nrad, nsec):
    d, f = _disk(nrad, nsec, nrad)
    for _ in range(2):
        g = d.fields()  # fresh arrays
        assert all(np.array_equal(f[k], g[k]) for k in FIELDS)
    out = {k: np.full((nrad + 1, nsec), -1, np.float32) for k in FIELDS}  # touched
    fp = C.POINTER(C.c_float)
    assert lib.fargo_download(d.ctx, *[out[k].ctypes.data_as(fp) for k in FIELDS], None, None) == 0
    assert all(np.array_equal(f[k], out[k]) for k in FIELDS)


def test_two_threads():
    pair = [_disk(800, 1200, 1), _disk(801, 1199, 2)]
    bad = []

    def run(d, f):
        for _ in range(20):
            g = d.fields()
            if not all(np.array_equal(f[k], g[k]) for k in FIELDS):
                bad.append(1)

    t = [threading.Thread(target=run, args=p) for p in pair]
    [x.start() for x in t]
    [x.join() for x in t]
    assert not bad
    for d, _ in pair:
        d.close()  # the ring goes with the last context, and a new one is made
    d, f = _disk(300, 1500, 3)
    assert np.array_equal(d.fields()["dens"], f["dens"])
