"""Determinant ratios of few walkers: blocks of fewer walkers, the same bits
as those walkers in a large population."""
import pytest

from einspline_gb300 import api


@pytest.mark.gpu
@pytest.mark.parametrize("storage", [api.STORE_F16, api.STORE_BF16])
@pytest.mark.parametrize("n", [1, 40, 129, 260])
def test_ratios_do_not_depend_on_the_population(storage, n):
    torch = pytest.importorskip("torch")
    G = api.MultiUBspline3D("s", [(0.0, 1.0, 7), (0.0, 1.0, 9), (0.0, 1.0, 8)], [(api.PERIODIC, api.PERIODIC)] * 3, n,
                            storage=storage)
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    G.set_device(0, torch.rand((n,) + G.M, device="cuda", generator=g) - 0.5)
    G.flush()
    W = 1700
    inv = torch.rand((W, n, n), device="cuda", generator=g) + 0.5
    pos = torch.rand((W, 3), device="cuda", generator=g)
    ref = api.Determinants(inv, inv, n).ratio(G, pos, n // 2)
    for w in (1, 2, 7, 8, 456, 457, 913, 1520, 1521):
        got = api.Determinants(inv[:w], inv[:w], n).ratio(G, pos[:w].contiguous(), n // 2)
        for a, b in zip(got, ref):
            assert torch.equal(a, b[:w]), w
