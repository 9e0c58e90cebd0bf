"""The boundary kernel where its sizes can go wrong, against the oracle: the
narrowest grid NONREFLECTING takes, a ring of one staged chunk and of one
chunk and a remainder (1024 and 1030 sectors), rows that are no multiple of
the block's four sectors a thread.  (The grids are fine enough for the
non-reflecting offsets to stay within a turn, as the reference needs.)  Substep counts, dt and
FARGO shifts exact; fields within twice the distance of the oracle's two FP32
builds (tests/helpers.py floor_tol, no less than its REF_TOL)."""
import numpy as np
import pytest

from tests.helpers import floor_tol
from tests.test_gpu_parity import _compare, _pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nrad,nsec,over", [
    ("adi", 32, 130, {"InnerBoundary": "NONREFLECTING"}),
    ("adi", 32, 1024, {"InnerBoundary": "NONREFLECTING"}),
    ("adi", 31, 1030, {"InnerBoundary": "NONREFLECTING"}),
    ("iso", 30, 517, {"InnerBoundary": "NONREFLECTING"}),
    ("iso", 16, 1025, {"InnerBoundary": "EVANESCENT", "Frame": "COROTATING"}),
    ("adi", 16, 255, {"InnerBoundary": "EVANESCENT"}),
    ("iso", 8, 131, {"InnerBoundary": "OPEN"})])
def test_boundary_sizes(gpu, kind, nrad, nsec, over):
    P, L, d, o, _ = _pair(kind, nrad, nsec, **over)
    start = {k: np.array(v) for k, v in d.fields().items()}
    n = d.advance_dt()
    assert n == o.advance_dt()
    keys = ("dens", "vrad", "vtheta") + (("energy",) if kind == "adi" else ())
    tol = floor_tol(P, L, start, 1, o.fields(), keys=keys)
    _compare(P, d, o, 0, fields=keys, tol=tol, planet_rtol=1e-5)
    assert np.array_equal(d.substep_log()[0], o.substep_log()[0])
    assert np.array_equal(d.substep_log()[1], o.substep_log()[1])
