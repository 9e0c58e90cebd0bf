"""NONREFLECTING on grids so coarse that an angular offset exceeds a turn: the
reference's one wrap then leads into another ring, and the sectors go in order,
as in the oracle (substep counts, dt and FARGO shifts exact, fields within
twice the distance of the oracle's two FP32 builds).  An offset whose target lies
outside the fields is refused, and so is a NaN in the edge rings' sound speed:
the DT ends with an error, the context stays usable and the same as a fresh one
from the same checkpoint."""
import numpy as np
import pytest

from cudaprotoplanetarydisksfloat_b200 import Disk, grid_radii, noise
from cudaprotoplanetarydisksfloat_b200._abi import FargoError
from tests.helpers import SEED, floor_tol, small
from tests.test_gpu_parity import _compare, _pair

pytestmark = pytest.mark.gpu


def _turns(P):
    """The initial state's offsets, in turns (locally isothermal sound speed, times sqrt(gamma))."""
    R = np.array(grid_radii(P), np.float64)
    Rm = 2 / 3 * (R[1:] ** 3 - R[:-1] ** 3) / (R[1:] ** 2 - R[:-1] ** 2)
    cs = P.ASPECTRATIO * Rm ** (P.FLARINGINDEX - 0.5) * (np.sqrt(P.ADIABATICINDEX) if P.Adiabatic else 1.0)
    inner = (R[1] ** -1.5 - 1) / (0.5 * (cs[0] + cs[1])) * (Rm[1] - Rm[0]) / (2 * np.pi)
    outer = (R[P.NRAD - 2] ** -1.5 - 1) / (0.5 * (cs[-1] + cs[-2])) * (Rm[-1] - Rm[-2]) / (2 * np.pi)
    return inner, outer


@pytest.mark.parametrize("kind,nrad,nsec", [("adi", 6, 517), ("adi", 12, 260), ("iso", 8, 131)])
def test_beyond_a_turn(gpu, kind, nrad, nsec):
    P, L, d, o, _ = _pair(kind, nrad, nsec, InnerBoundary="NONREFLECTING", DT="0.1")
    assert 1.02 < max(abs(t) for t in _turns(P)) < 2.0
    start = {k: np.array(v) for k, v in d.fields().items()}
    assert d.advance_dt() == o.advance_dt()
    keys = ("dens", "vrad", "vtheta") + (("energy",) if kind == "adi" else ())
    tol = floor_tol(P, L, start, 1, o.fields(), keys=keys)
    _compare(P, d, o, 0, fields=keys, tol=tol, planet_rtol=1e-5)
    assert np.array_equal(d.substep_log()[0], o.substep_log()[0])
    assert np.array_equal(d.substep_log()[1], o.substep_log()[1])


def _usable(P, L, d, blob):
    d.restore(blob)
    e = Disk(P, L)
    e.restore(blob)
    assert d.advance_dt() == e.advance_dt() > 0
    f, g = d.fields(), e.fields()
    for k in f:
        assert np.array_equal(f[k], g[k]), k


@pytest.mark.parametrize("graph", [True, False])
def test_outside_the_fields_is_refused(gpu, graph):
    P, L, _ = small("adi", 8, 130, InnerBoundary="NONREFLECTING", AspectRatio="0.01")
    assert _turns(P)[1] < -4.0
    d = Disk(P, L)
    d.set_graph_mode(graph)
    for _ in range(2):
        with pytest.raises(FargoError, match="EINVAL"):
            d.advance_dt()
        assert d.scalars()["nsub_last_dt"] == 1


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("ring", [0, 1, 30, 31])
def test_nan_at_the_edge(gpu, graph, ring):
    P, L, _ = small("adi", 32, 130, InnerBoundary="NONREFLECTING")
    d = Disk(P, L)
    d.set_graph_mode(graph)
    d.init_state(dens=noise.perturb_density(d.fields()["dens"].reshape(-1), 32, 130, SEED))
    blob = d.checkpoint()
    e = d.fields()["energy"].copy()
    e[ring, 5] = np.nan
    d.upload(energy=e)
    with pytest.raises(FargoError, match="ENONFINITE"):
        d.advance_dt()
    _usable(P, L, d, blob)
