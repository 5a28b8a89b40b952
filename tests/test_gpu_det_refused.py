"""Where a refused update (a walker index out of range in a CUDA tensor) shows:
in check_updates, and in the next ratio or update; once."""
import pytest

from einspline_gb300 import api

N, W, K = 5, 3, 2


def population(torch):
    A = torch.eye(N, device="cuda").repeat(W, 1, 1)
    return api.Determinants(A, A.clone(), N), A[:, K] + 0.1


def table(torch):
    G = api.MultiUBspline3D("s", [(0.0, 1.0, 6)] * 3, [(api.PERIODIC, api.PERIODIC)] * 3, N)
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    G.set_device(0, torch.rand((N, 6, 6, 6), device="cuda", generator=g))
    G.flush()
    return G


@pytest.mark.gpu
def test_ratio_reports_a_refused_update():
    torch = pytest.importorskip("torch")
    D, rows = population(torch)
    G = table(torch)
    pos = torch.rand((W, 3), device="cuda")
    before = D.ratio(G, pos, K)[0]
    D.update(K, torch.tensor([0, W], device="cuda"), rows)
    torch.cuda.synchronize()
    with pytest.raises(IndexError):
        D.ratio(G, pos, K)
    assert torch.equal(D.ratio(G, pos, K)[0], before)


@pytest.mark.gpu
def test_check_updates_reports_once():
    torch = pytest.importorskip("torch")
    D, rows = population(torch)
    D.check_updates()
    D.update(K, torch.tensor([-W - 1], device="cuda"), rows)
    torch.cuda.synchronize()
    with pytest.raises(IndexError):
        D.check_updates()
    D.check_updates()
    D.update(K, torch.tensor([-W], device="cuda"), rows)
    torch.cuda.synchronize()
    D.check_updates()
    assert torch.equal(D.A[0, K], rows[0])


@pytest.mark.gpu
def test_a_late_refusal_is_not_the_next_objects():
    """A launch that is still pending when its object goes, and is refused
    then, says nothing about an object made since."""
    torch = pytest.importorskip("torch")
    big = torch.zeros(256 << 20, device="cuda")
    bad, good = torch.tensor([W], device="cuda"), torch.tensor([0], device="cuda")
    D, rows = population(torch)
    D.update(K, good, rows)
    torch.cuda.synchronize()
    done = torch.cuda.Event()
    for _ in range(100):
        big.add_(1.0)  # tens of milliseconds in front of the refusal
    D.update(K, bad, rows)
    done.record()
    del D
    others = [population(torch)[0] for _ in range(3)]
    assert not done.query()
    torch.cuda.synchronize()
    for E in others:
        E.check_updates()
    others[0].update(K, bad, rows)
    torch.cuda.synchronize()
    others[1].check_updates()
    with pytest.raises(IndexError):
        others[0].check_updates()
