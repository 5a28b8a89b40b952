"""Determinants.update by walker index: any order, negative indices and index
types give the bits of the same walkers in a call of their own, other walkers
keep theirs, and an index out of range refuses the whole call."""
import pytest

from einspline_gb300 import api


def population(torch, W, n, trans):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    A = torch.eye(n, device="cuda") + 0.3 / n ** 0.5 * torch.randn((W, n, n), device="cuda", generator=g)
    inv = torch.linalg.inv(A.double()).float()
    inv = (inv.transpose(1, 2) if trans else inv).contiguous()
    rows = A[:, n // 2] + 0.1 / n ** 0.5 * torch.randn((W, n), device="cuda", generator=g)
    return A, inv, rows.contiguous()


@pytest.mark.gpu
@pytest.mark.parametrize("trans", [0, 1])
@pytest.mark.parametrize("n,W", [(5, 1), (64, 40), (33, 1500), (2052, 3)])
def test_accepted_walkers(n, W, trans):
    torch = pytest.importorskip("torch")
    A, inv, rows = population(torch, W, n, trans)
    refA, refI = A.clone(), inv.clone()
    api.Determinants(refA, refI, n, trans).update(n // 2, torch.arange(W, device="cuda"), rows)
    order = torch.randperm(W, device="cuda")[:max(1, 2 * W // 3)]
    chosen = torch.zeros(W, dtype=torch.bool, device="cuda")
    chosen[order] = True
    for idx in (order, order.int(), order - W, order.tolist()):
        a, b = A.clone(), inv.clone()
        api.Determinants(a, b, n, trans).update(n // 2, idx, rows)
        for got, ref, old in ((a, refA, A), (b, refI, inv)):
            assert torch.equal(got[chosen], ref[chosen])
            assert torch.equal(got[~chosen], old[~chosen])


@pytest.mark.gpu
@pytest.mark.parametrize("n,W,bad", [(64, 40, 40), (64, 40, -41), (2052, 3, 7)])
def test_index_out_of_range_updates_nothing(n, W, bad):
    torch = pytest.importorskip("torch")
    A, inv, rows = population(torch, W, n, 0)
    a, b = A.clone(), inv.clone()
    D = api.Determinants(a, b, n, 0)
    D.update(n // 2, torch.tensor([0, bad, 1], device="cuda"), rows)
    torch.cuda.synchronize()
    assert torch.equal(a, A) and torch.equal(b, inv)
    with pytest.raises(IndexError):
        D.update(n // 2, [0], rows)
    D.update(n // 2, [0], rows)
    assert torch.equal(a[0, n // 2], rows[0]) and torch.equal(b[1:], inv[1:])
