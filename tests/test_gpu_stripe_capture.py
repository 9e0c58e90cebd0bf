"""The stripe calls under a caller's capture of the stripe's stream: whatever the
caller captures next must come after every kernel of the substep, so the captured
nodes form one chain with a single last node (the library's own graph has side
branches).  The graph is looked at, not run."""
import ctypes as C

import pytest
import torch

from cudaprotoplanetarydisksfloat_b200 import radial
from cudaprotoplanetarydisksfloat_b200._abi import lib
from tests.helpers import small

pytestmark = pytest.mark.gpu


def _last_nodes(rt, graph):
    n = C.c_size_t(0)
    assert rt.cudaGraphGetNodes(graph, None, C.byref(n)) == 0
    nodes = (C.c_void_p * n.value)()
    assert rt.cudaGraphGetNodes(graph, nodes, C.byref(n)) == 0
    m = C.c_size_t(0)
    assert rt.cudaGraphGetEdges_v2(graph, None, None, None, C.byref(m)) == 0
    a, b, data = (C.c_void_p * m.value)(), (C.c_void_p * m.value)(), (C.c_uint64 * m.value)()
    assert rt.cudaGraphGetEdges_v2(graph, a, b, data, C.byref(m)) == 0
    return len(nodes), set(nodes) - set(a)


@pytest.mark.parametrize("kind", ["iso", "adi"])
def test_one_last_node(gpu, kind):
    P, L, _ = small(kind, 64, 128)
    st = radial.LocalStripes(P, L, 2)
    s = st.stripes[0]
    blocks = torch.zeros(2 * s.stride, dtype=torch.float64, device=s.device)
    rt = C.CDLL("libcudart.so.12")
    stream, graph = C.c_void_p(s.stream.cuda_stream), C.c_void_p()
    torch.cuda.synchronize()
    assert rt.cudaStreamBeginCapture(stream, 1) == 0  # thread-local mode
    e0 = lib.fargo_stripe_substep(s.ctx, C.c_void_p(blocks.data_ptr()), 2, s.stride)
    e1 = lib.fargo_stripe_forces(s.ctx, C.c_void_p(s.block.data_ptr()))
    assert rt.cudaStreamEndCapture(stream, C.byref(graph)) == 0
    assert e0 == 0 and e1 == 0
    n, last = _last_nodes(rt, graph)
    assert n > 8 and len(last) == 1, (n, len(last))
    rt.cudaGraphDestroy(graph)
