"""Determinants.update on a stream other than the current one: the order in
which memory and indices reach that stream."""
import contextlib

import pytest

from einspline_gb300 import api


class Recorder:
    """Stands in for the library and for torch's streams, without a GPU."""

    def __init__(self, torch, monkeypatch):
        self.log, self.at = [], "current"
        empty = torch.empty

        def logged_empty(*a, **k):
            self.log.append(("alloc", self.at))
            return empty(*a, **k)

        @contextlib.contextmanager
        def on(stream):
            self.at, before = stream, self.at
            yield
            self.at = before

        monkeypatch.setattr(torch, "empty", logged_empty)
        monkeypatch.setattr(torch.cuda, "stream", on)
        monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: "current")
        monkeypatch.setattr(torch.cuda, "Stream", Recorder)
        monkeypatch.setattr(torch.Tensor, "record_stream", lambda t, s: self.log.append(("keep", t.data_ptr(), s)))
        monkeypatch.setattr(api, "_lib", lambda: self)

    def wait_stream(self, other):
        self.log.append(("wait", other))

    cuda_stream = 7

    def einspline_gb300_det_update_accepted_mark(self, o, n, idx, batch, work, scratch, status, mark, stream):
        self.log.append(("launch", idx, work, stream))
        return 0


@pytest.mark.parametrize("kind", ["int64", "int32", "list"])
def test_update_on_another_stream_is_ordered(monkeypatch, kind):
    torch = pytest.importorskip("torch")
    A = torch.eye(4).repeat(3, 1, 1)
    rows = A[:, 1].contiguous()
    D = api.Determinants(A, A.clone(), 4)
    s = Recorder(torch, monkeypatch)
    idx = [0, 2] if kind == "list" else torch.tensor([0, 2], dtype=getattr(torch, kind))
    D.update(1, idx, rows, stream=s)
    (launch,) = [e for e in s.log if e[0] == "launch"]
    before = s.log[:s.log.index(launch)]
    assert launch[3] == 7
    # scratch comes from the stream's memory, not from memory that the
    # current stream may still be using
    assert [e for e in before if e[0] == "alloc"] == [("alloc", s)]
    # indices that the current stream makes are waited for
    assert (("wait", "current") in before) == (kind != "list")
    # indices and work space stay until the stream is done with them
    assert ("keep", launch[1], s) in s.log and ("keep", launch[2], s) in s.log


def test_stream_of_another_library(monkeypatch):
    """An object with a cuda_stream handle is a stream, as for the other calls."""
    torch = pytest.importorskip("torch")
    A = torch.eye(4).repeat(3, 1, 1)
    rows = A[:, 1].contiguous()
    D = api.Determinants(A, A.clone(), 4)
    s = Recorder(torch, monkeypatch)
    s.cuda_stream = 11
    monkeypatch.setattr(torch.cuda, "ExternalStream", lambda handle: s if handle == 11 else None)
    foreign = type("Foreign", (), {"cuda_stream": 11})()
    D.update(1, [0, 2], rows, stream=foreign)
    (launch,) = [e for e in s.log if e[0] == "launch"]
    assert launch[3] == 11 and ("alloc", s) in s.log and ("keep", launch[1], s) in s.log


@pytest.mark.gpu
@pytest.mark.parametrize("trans", [0, 1])
def test_update_beside_a_busy_current_stream(trans):
    torch = pytest.importorskip("torch")
    W, n, k = 64, 33, 5
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    A = torch.eye(n, device="cuda") + 0.05 * torch.randn((W, n, n), device="cuda", generator=g)
    inv = torch.linalg.inv(A.double()).float()
    inv = (inv.transpose(1, 2) if trans else inv).contiguous()
    rows = A[:, k] + 0.01
    order = torch.randperm(W, device="cuda")[:40]
    refA, refI = A.clone(), inv.clone()
    api.Determinants(refA, refI, n, trans).update(k, order, rows)
    side = torch.cuda.Stream()
    big = torch.zeros(64 << 20, device="cuda")
    for idx in (order, order.int(), order.tolist()):
        a, b = A.clone(), inv.clone()
        D = api.Determinants(a, b, n, trans)
        torch.cuda.synchronize()
        for _ in range(8):
            big.add_(1.0)  # keeps the current stream busy
        for _ in range(4):  # blocks of the scratch's size, freed with writes to them pending
            torch.full((3 * 40 + 1,), -1, dtype=torch.int64, device="cuda")
        D.update(k, idx + 0 if torch.is_tensor(idx) else idx, rows, stream=side)
        for _ in range(4):
            torch.full((3 * 40 + 1,), -1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        assert torch.equal(a, refA) and torch.equal(b, refI)
