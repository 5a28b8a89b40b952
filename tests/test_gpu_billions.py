"""FP32 values of a few columns at billions of points in one call.  The launch
is captured into a graph that never runs, so it needs no memory for them."""
import ctypes as C

import pytest

from einspline_gb300 import api


@pytest.mark.gpu
# a table between L2's size and what goes in cell order (one point a block), and one that L2 holds
@pytest.mark.parametrize("g,npts", [(104, 2 ** 31 + 5), (8, 2 ** 33 + 9)])
@pytest.mark.parametrize("N", [1, 5])
def test_one_call_of_billions_of_points(g, npts, N):
    torch = pytest.importorskip("torch")
    G = api.MultiUBspline3D("s", [(0.0, 1.0, g)] * 3, [(api.PERIODIC, api.PERIODIC)] * 3, N)
    pos = torch.zeros((4, 3), device="cuda")
    out = torch.zeros((4, N), device="cuda")
    G.eval(pos, vgh=False, out=(out, None, None))  # first use outside the capture
    torch.cuda.synchronize()
    o = G.opts(False, False, 1, 0, False)
    graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=s):
        r = api._lib().einspline_gb300_eval_3d(G.table, C.byref(o), npts, pos.data_ptr(), out.data_ptr(), None, None,
                                               s.cuda_stream)
    del graph
    assert r == 0
