"""The planets' branch of the substep graph: beside the gas kernels in a fixed
frame, before them in a corotating one, in line in the host loop.  The two
forms run the same kernels, so they give the same bits; and the parity tests
check the results against the oracle."""
import numpy as np
import pytest

from cudaprotoplanetarydisksfloat_b200 import Disk, noise, planets_dict
from tests.helpers import SEED, make, small
from cudaprotoplanetarydisksfloat_b200 import configs

pytestmark = pytest.mark.gpu


def _run(P, L, graph, ndt=2):
    d = Disk(P, L)
    d.set_graph_mode(graph)
    f0 = d.fields()
    d.init_state(dens=noise.perturb_density(f0["dens"].reshape(-1), P.NRAD, P.NSEC, SEED))
    n = [d.advance_dt() for _ in range(ndt)]
    out = dict(d.fields(), nsub=np.array(n), **planets_dict(d.planets()))
    d.close()
    return out


# 17 planets: the integrator's scratch no longer fits in shared memory
@pytest.mark.parametrize("kind,over,extra", [
    ("adi", {}, 0), ("adi", {"Frame": "COROTATING"}, 0), ("iso", {"Frame": "GUIDING-CENTER"}, 0),
    ("iso", {}, 16), ("adi", {"Disk": "NO"}, 0)])
def test_graph_and_host_loop_agree(kind, over, extra):
    if extra:
        p, pl = configs.small(kind, 32, 96)
        p = dict(p, ForcedCircular="NO")
        pl = [pl[0][:3] + ("YES", "YES")] + [("Q%c" % (65 + k), 0.6 + 0.1 * k, 1e-7, "NO", "YES") for k in range(extra)]
        P, L, _ = make(p, pl, "many")
    else:
        P, L, _ = small(kind, 32, 96, **over)
    a, b = _run(P, L, True), _run(P, L, False)
    for k in a:
        assert np.array_equal(a[k], b[k]), k
