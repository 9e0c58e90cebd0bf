"""Field downloads around the size from which touched destinations go through
the copy ring (24 MiB): one grid just below it and two above, exact into fresh,
touched and page-locked destinations."""
import ctypes as C

import numpy as np
import pytest
import torch

from cudaprotoplanetarydisksfloat_b200._abi import lib
from tests.test_gpu_host_copy import FIELDS, _disk

pytestmark = pytest.mark.gpu

LIMIT = 24 << 20


@pytest.mark.parametrize("nrad,nsec,above", [(1200, 1301, False), (1300, 1301, True), (1700, 2047, True)])
def test_touched_and_page_locked(gpu, nrad, nsec, above):
    assert (4 * 4 * (nrad + 1) * nsec >= LIMIT) == above
    d, f = _disk(nrad, nsec, nrad)
    fp = C.POINTER(C.c_float)

    def check(out):
        assert lib.fargo_download(d.ctx, *[out[k].ctypes.data_as(fp) for k in FIELDS], None, None) == 0
        assert all(np.array_equal(f[k], out[k]) for k in FIELDS)

    assert all(np.array_equal(f[k], v) for k, v in d.fields().items())
    locked = {k: torch.full((nrad + 1, nsec), -1.0).pin_memory() for k in FIELDS}
    for _ in range(2):
        check({k: np.full((nrad + 1, nsec), -1, np.float32) for k in FIELDS})
        check({k: v.numpy() for k, v in locked.items()})
        # one page-locked among pageable ones
        mixed = {k: np.full((nrad + 1, nsec), -1, np.float32) for k in FIELDS}
        locked["vrad"].fill_(-1)
        check(dict(mixed, vrad=locked["vrad"].numpy()))
    d.close()
