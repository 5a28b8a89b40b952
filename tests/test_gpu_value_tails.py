"""Values of 16-bit tables whose columns leave a ragged last tile: the wide
copy pipeline deals those columns to all lanes of its warps.  Bit-identical to
the direct-load kernel, whose threads keep to one column group."""
import pytest

from einspline_gb300 import api

GRID = [(0.0, 1.0, 9), (-1.0, 1.0, 8), (0.0, 2.0, 10)]
PER = [(api.PERIODIC, api.PERIODIC)] * 3


@pytest.mark.gpu
@pytest.mark.parametrize("storage", [api.STORE_I16, api.STORE_F16, api.STORE_BF16])
@pytest.mark.parametrize("cols", [1, 8, 9, 100, 255, 256, 257, 384, 505, 777])
def test_ragged_last_tile(storage, cols):
    torch = pytest.importorskip("torch")
    G = api.MultiUBspline3D("s", GRID, PER, cols, storage=storage)
    g = torch.Generator(device="cuda")
    g.manual_seed(cols)
    G.set_device(0, torch.rand((cols,) + G.M, generator=g, device="cuda") - 0.5)
    G.flush()
    pos = torch.rand((5003, 3), generator=g, device="cuda", dtype=torch.float64)
    G.set_load_mode(0)
    ref = G.eval(pos, vgh=False)[0]
    G.set_load_mode(3)
    for n in (1, 2, 3, 15, 16, 17, 31, 33, 200, 5003):
        out = torch.full((n, ref.shape[1]), float("nan"), device="cuda")
        G.eval(pos[:n], vgh=False, out=(out, None, None))
        assert torch.equal(out, ref[:n]), n
