"""Output rows that start off a 16-byte boundary: an odd number of splines or
a buffer at any element.  Bit-identical to the aligned rows of a table whose
first splines are the same, and nothing outside the rows is written."""
import pytest

from einspline_gb300 import api

GRID = [(0.0, 1.0, 8), (-1.0, 1.0, 7), (0.0, 2.0, 9)]
PER = [(api.PERIODIC, api.PERIODIC)] * 3
GRID_M = tuple(n for _, _, n in GRID)  # periodic: one datum a cell


def table(torch, kind, storage, data):
    G = api.MultiUBspline3D(kind, GRID, PER, data.shape[0], storage=storage)
    G.set_device(0, data)
    G.flush()
    return G


@pytest.mark.gpu
@pytest.mark.parametrize("kind,storage,modes", [("s", 0, (0, 2, 4)), ("s", api.STORE_I16, (0, 2, 3, 4)),
                                                ("s", api.STORE_BF16, (3, 5)), ("c", 0, (0, 2)),
                                                ("c", api.STORE_F16, (3, 5))])
@pytest.mark.parametrize("N", [1, 2, 3, 31, 33, 127, 130, 203, 257])
def test_shifted_rows(kind, storage, modes, N):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    P = 301
    pos = torch.rand((P, 3), generator=g, device="cuda", dtype=torch.float64)
    shape = ((N + 7) // 4 * 4,) + GRID_M + ((2,) if kind == "c" else ())
    data = torch.rand(shape, generator=g, device="cuda") - 0.5
    G, R = table(torch, kind, storage, data[:N].contiguous()), table(torch, kind, storage, data)
    for mode in modes:
        G.set_load_mode(mode)
        R.set_load_mode(mode)
        for layout in (0, 1):
            ref = R.eval(pos, layout=layout)
            for off in range(4):
                buf = [torch.full((16 + torch.Size(s).numel(),), float("nan"), device="cuda")
                       for s in G.out_shapes(P, layout)]
                out = tuple(b[4 + off:4 + off + b.numel() - 16].view(s) for b, s in zip(buf, G.out_shapes(P, layout)))
                G.eval(pos, layout=layout, out=out)
                for b, a, r in zip(buf, out, ref):
                    assert torch.equal(a, r[:, :N]), (mode, layout, off)
                    assert torch.isnan(b[:4 + off]).all() and torch.isnan(b[off - 12:]).all(), (mode, layout, off)
