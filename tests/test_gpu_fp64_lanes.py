"""FP64 vgh with fewer columns than a block has threads: its (point, columns)
pairs are dealt to all threads, in blocks sized by the batch.  The same bits
as launches whose shape gives every point a row of threads."""
import pytest

from einspline_gb300 import api

GRID = [(0.0, 1.0, 9), (-1.0, 1.0, 7), (0.0, 2.0, 8)]


@pytest.mark.gpu
@pytest.mark.parametrize("kind,N", [("d", 1), ("d", 2), ("d", 5), ("z", 8), ("d", 63), ("d", 64), ("d", 65),
                                    ("d", 203), ("z", 129), ("d", 260)])
def test_dealt_columns(kind, N):
    torch = pytest.importorskip("torch")
    G = api.MultiUBspline3D(kind, GRID, [(api.PERIODIC, api.PERIODIC)] * 3, N)
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    G.set_device(0, torch.rand((N,) + G.M + ((2,) if kind == "z" else ()), generator=g, device="cuda",
                               dtype=torch.float64) - 0.5)
    G.flush()
    pos = torch.rand((9001, 3), generator=g, device="cuda", dtype=torch.float64)
    ref = G.eval(pos)  # 9001 points one by one cover every lane of the walk
    one = [G.eval(pos[i:i + 1]) for i in (0, 1, 17, 4500, 9000)]
    for j, i in enumerate((0, 1, 17, 4500, 9000)):
        for a, b in zip(one[j], ref):
            assert torch.equal(a[0], b[i]), i
    for layout in (0, 1):
        ref = G.eval(pos, layout=layout)
        for n in (2, 3, 15, 16, 17, 63, 64, 65, 300, 1537, 3001):
            for a, b in zip(G.eval(pos[:n], layout=layout), ref):
                assert torch.equal(a, b[:n]), (layout, n)
    ref = G.eval(pos)
    for tx, ty, pb in ((32, 1, 1), (32, 8, 16), (64, 2, 7), (128, 1, 64), (256, 1, 3)):
        G.set_tile(tx, ty, pb)
        for a, b in zip(G.eval(pos), ref):
            assert torch.equal(a, b), (tx, ty, pb)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,N", [("d", 1), ("d", 3), ("z", 8), ("d", 64), ("d", 203), ("z", 257)])
def test_dealt_values(kind, N):
    torch = pytest.importorskip("torch")
    G = api.MultiUBspline3D(kind, GRID, [(api.PERIODIC, api.PERIODIC)] * 3, N)
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    G.set_device(0, torch.rand((N,) + G.M + ((2,) if kind == "z" else ()), generator=g, device="cuda",
                               dtype=torch.float64) - 0.5)
    G.flush()
    pos = torch.rand((9001, 3), generator=g, device="cuda", dtype=torch.float64)
    ref = G.eval(pos, vgh=False)[0]
    assert torch.equal(ref, G.eval(pos)[0])
    for n in (1, 2, 17, 64, 65, 300, 3001):
        assert torch.equal(G.eval(pos[:n], vgh=False)[0], ref[:n]), n
