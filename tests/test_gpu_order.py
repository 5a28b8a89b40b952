"""Large batches on large tables are put into cell order by the library
(launch_eval_ordered): bit for bit the results of the same points in batches
small enough to keep their order, for every form an entry takes, from several
streams at once, and not under stream capture."""
import ctypes as C

import numpy as np
import pytest

from einspline_gb300 import _lib as L
from einspline_gb300 import api

GRID = [(0.0, 1.0, 60), (0.0, 1.0, 64), (0.0, 1.0, 56)]
PER = [(api.PERIODIC, api.PERIODIC)] * 3
SMALL = 1500  # points a batch that stays in its order
_tables = {}


def table(torch, kind, storage, N):
    key = (kind, storage, N)
    if key not in _tables:
        _tables.clear()  # one at a time
        G = api.MultiUBspline3D(kind, GRID, PER, N, storage=storage)
        g = torch.Generator(device="cuda")
        g.manual_seed(N)
        shape = (N,) + G.M + ((2,) if kind in "cz" else ())
        G.set_device(0, torch.rand(shape, generator=g, device="cuda",
                                   dtype=torch.float32 if kind in "sc" else torch.float64) - 0.5)
        G.flush()
        assert G.info().table_bytes > 192 << 20
        _tables[key] = G
    return _tables[key]


def points(torch, n, dt, seed=1):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.rand((n, 3), generator=g, device="cuda", dtype=dt) * 1.02 - 0.01  # some outside the box


def launches(f):
    n0 = api.launch_count()
    r = f()
    return r, api.launch_count() - n0


FORMS = [("s", api.STORE_NATIVE, 513), ("s", api.STORE_F16, 1000), ("s", api.STORE_BF16, 1000),
         ("s", api.STORE_I16, 1000), ("c", api.STORE_NATIVE, 255), ("c", api.STORE_F16, 500)]


@pytest.mark.gpu
@pytest.mark.parametrize("kind,storage,N", FORMS)
def test_flat_entry(kind, storage, N):
    torch = pytest.importorskip("torch")
    G = table(torch, kind, storage, N)
    n = 12000 if storage != api.STORE_I16 else 24000
    for dt, rule, layout, vgh in ((torch.float64, 0, 0, True), (torch.float32, 1, 1, True), (torch.float64, 1, 0, False)):
        pos = points(torch, n, dt)
        got, count = launches(lambda: G.eval(pos, vgh=vgh, rule=rule, layout=layout))
        assert count == 3  # two sort launches and the evaluation
        for p0 in range(0, n, SMALL):
            ref, count = launches(lambda: G.eval(pos[p0:p0 + SMALL], vgh=vgh, rule=rule, layout=layout))
            assert count == 1
            for a, b in zip(got, ref):
                if b is not None:
                    assert torch.equal(a[p0:p0 + SMALL], b), (dt, rule, layout, vgh, p0)


@pytest.mark.gpu
def test_strided_outputs_and_several_windows():
    """Batches beyond one sort's points go window by window."""
    torch = pytest.importorskip("torch")
    G = table(torch, "s", api.STORE_F16, 1000)
    N, n = 1000, 131072 + 9001
    pos = points(torch, n, torch.float64)
    vs = N + 7
    out = torch.full((n, vs), 5.0, device="cuda")
    o = G.opts(False, True, 0, 0, False, (vs, 0, 0))

    def call(p0, p1):
        L.load().einspline_gb300_eval_3d(G.table, C.byref(o), p1 - p0, C.c_void_p(pos[p0:].data_ptr()),
                                         C.c_void_p(out[p0:].data_ptr()), None, None,
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream))
        L.check()
    _, count = launches(lambda: call(0, n))
    assert count == 6
    got = out.clone()
    out.fill_(5.0)
    for p0 in range(0, n, SMALL):
        call(p0, min(n, p0 + SMALL))
    assert torch.equal(got, out)


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["vgh", "value", "vgl", "vgl_sign", "sign"])
def test_pointer_entries(form):
    torch = pytest.importorskip("torch")
    G = table(torch, "s", api.STORE_NATIVE, 513)
    H = G.to_cuda()
    n = 12000
    pos = points(torch, n, torch.float32)
    sign = torch.where(torch.arange(n, device="cuda") % 3 == 0, -1.0, 1.0)
    linv = torch.tensor([1.1, 0.1, 0.0, 0.2, 0.9, -0.1, 0.0, 0.3, 1.2], device="cuda")

    def call(p, s):
        if form == "vgh":
            return H.eval_multi(p)
        if form == "value":
            return H.eval_multi(p, vgh=False)[:1]
        if form == "sign":
            return (H.eval_multi_sign(p, s),)
        return H.eval_multi_vgl(p, linv, row_stride=520, sign=s if form == "vgl_sign" else None)
    got, count = launches(lambda: call(pos, sign))
    assert count == 3
    for p0 in range(0, n, SMALL):
        ref, count = launches(lambda: call(pos[p0:p0 + SMALL].contiguous(), sign[p0:p0 + SMALL].contiguous()))
        assert count == 1
        for a, b in zip(got, ref):
            assert torch.equal(a[p0:p0 + SMALL], b), p0
    H.destroy()


@pytest.mark.gpu
def test_streams_and_capture():
    """More streams than pieces of scratch, their launches in flight together,
    then streams that come and go; a captured launch keeps its order."""
    torch = pytest.importorskip("torch")
    G = table(torch, "s", api.STORE_F16, 1000)
    pos = [points(torch, 9000 + 700 * k, torch.float64, seed=k) for k in range(7)]
    ref = [[x.clone() for x in G.eval(p)] for p in pos]
    torch.cuda.synchronize()
    for rep in range(3):
        streams = [torch.cuda.Stream() for _ in pos]
        outs = []
        for _ in range(2):
            for p, s in zip(pos, streams):
                with torch.cuda.stream(s):
                    outs.append(G.eval(p, stream=s))
        torch.cuda.synchronize()
        for i, o in enumerate(outs):
            for a, b in zip(o, ref[i % len(pos)]):
                assert torch.equal(a, b), (rep, i)
        del outs
    out = tuple(torch.zeros_like(x) for x in ref[0])
    graph = torch.cuda.CUDAGraph()
    n0 = api.launch_count()
    with torch.cuda.graph(graph):
        G.eval(pos[0], out=out)
    assert api.launch_count() - n0 == 1
    graph.replay()
    got = [x.clone() for x in G.eval(pos[1])]
    graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(out, ref[0]):
        assert torch.equal(a, b)
    for a, b in zip(got, ref[1]):
        assert torch.equal(a, b)


@pytest.mark.gpu
def test_fp64_tables_keep_their_order():
    torch = pytest.importorskip("torch")
    G = table(torch, "d", api.STORE_NATIVE, 256)
    pos = points(torch, 12000, torch.float64)
    for mode, vgh, n in ((0, True, 1), (0, False, 1), (1, True, 1), (1, False, 3)):
        G.set_fp64_mode(mode)
        got, count = launches(lambda: G.eval(pos, vgh=vgh))
        assert count == n
        for p0 in range(0, 12000, 3 * SMALL):
            for a, b in zip(got, G.eval(pos[p0:p0 + 3 * SMALL], vgh=vgh)):
                if b is not None:
                    assert torch.equal(a[p0:p0 + 3 * SMALL], b)
    _tables.clear()


@pytest.mark.gpu
@pytest.mark.parametrize("kind,storage,vgh", [("s", api.STORE_NATIVE, False), ("s", api.STORE_F16, True),
                                              ("s", api.STORE_NATIVE, True), ("d", api.STORE_NATIVE, False)])
@pytest.mark.parametrize("n", [131072, 131073, 262144])
def test_large_sorted_batches(kind, storage, vgh, n):
    """Around the size where values of FP32 tables turn to the radix sort and
    everything else goes on with the counting sort: both sorted entries give
    the unsorted bits."""
    torch = pytest.importorskip("torch")
    G = api.MultiUBspline3D(kind, [(0.0, 1.0, 33), (0.0, 1.0, 9), (0.0, 1.0, 20)], PER, 6, storage=storage)
    dt = torch.float32 if kind == "s" else torch.float64
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    G.set_device(0, torch.rand((6,) + G.M, generator=g, device="cuda", dtype=dt) - 0.5)
    pos = points(torch, n, torch.float64)
    ref = G.eval(pos, vgh=vgh)
    got = G.eval(pos, vgh=vgh, sort=True)
    out = [torch.full_like(x, 3.0) if x is not None else None for x in ref]
    o = G.opts(vgh, True, 0, 0, True)
    p = lambda t: C.c_void_p(t.data_ptr() if t is not None else 0)  # noqa: E731
    L.load().einspline_gb300_eval_3d_sorted_noalloc(G.table, C.byref(o), n, p(pos), p(out[0]), p(out[1]), p(out[2]),
                                                    C.c_void_p(torch.cuda.current_stream().cuda_stream))
    L.check()
    for a, b, c in zip(ref, got, out):
        if a is not None:
            assert torch.equal(a, b) and torch.equal(a, c)
