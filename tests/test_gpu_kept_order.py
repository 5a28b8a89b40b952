"""sort = -1: a large batch on a large table keeps the caller's order (one
launch, no ordering in front of it) with the same bits."""
import pytest

from einspline_gb300 import api


@pytest.mark.gpu
@pytest.mark.parametrize("storage", [api.STORE_NATIVE, api.STORE_F16])
@pytest.mark.parametrize("vgh", [False, True])
def test_order_is_kept(storage, vgh):
    torch = pytest.importorskip("torch")
    N, P = 1000 if storage == api.STORE_F16 else 513, 20000
    G = api.MultiUBspline3D("s", [(0.0, 1.0, 60)] * 3, [(api.PERIODIC, api.PERIODIC)] * 3, N, storage=storage)
    g = torch.Generator(device="cuda")
    g.manual_seed(2)
    G.set_device(0, torch.rand((N, 60, 60, 60), device="cuda", generator=g))
    G.flush()
    pos = torch.rand((P, 3), device="cuda", generator=g)

    def launches(sort, p):
        n0 = api.launch_count()
        out = G.eval(p, vgh=vgh, sort=sort)
        return out, api.launch_count() - n0

    ordered, n_ordered = launches(False, pos)
    kept, n_kept = launches(-1, pos)
    assert (n_ordered, n_kept) == (3, 1)
    for a, b in zip(ordered, kept):
        assert a is None or torch.equal(a, b)
    assert launches(-1, pos[:1])[1] == 1
