"""Determinants over host tensors: the object works as far as no kernel runs."""
import pytest

from einspline_gb300 import api


def population(torch, W=3, n=4):
    A = torch.eye(n).repeat(W, 1, 1)
    return api.Determinants(A, A.clone(), n), A[:, 1].contiguous()


@pytest.mark.parametrize("none", [[], ()])
def test_no_accepted_walker_updates_nothing(none):
    torch = pytest.importorskip("torch")
    D, rows = population(torch)
    assert D.update(1, none, rows) is None
    assert D.update(1, torch.zeros(0, dtype=torch.int32), rows) is None


def test_update_reaches_the_library(monkeypatch):
    torch = pytest.importorskip("torch")
    D, rows = population(torch)

    class Lib:
        def einspline_gb300_det_update_accepted_mark(self, o, n, idx, batch, work, scratch, status, mark, stream):
            assert n == 2 and idx and work and scratch and not status and stream == 5
            return 0

    monkeypatch.setattr(api, "_lib", Lib)
    monkeypatch.setattr(api, "_stream", lambda torch, stream: 5)
    D.update(1, [0, 2], rows)


def test_rows_of_another_device_are_refused(monkeypatch):
    """Their addresses would otherwise reach a kernel of the matrices' device."""
    torch = pytest.importorskip("torch")
    D, _ = population(torch)
    called = []
    monkeypatch.setattr(api, "_lib", lambda: called.append(1))
    monkeypatch.setattr(api, "_stream", lambda torch, stream: 5)
    with pytest.raises(RuntimeError):
        D.update(1, [0, 2], torch.empty((3, 4), device="meta"))
    assert not called


@pytest.mark.parametrize("bad", [3, -4])
@pytest.mark.parametrize("make", ["list", "int64", "int32"])
def test_index_known_to_the_host_is_checked_at_once(monkeypatch, bad, make):
    torch = pytest.importorskip("torch")
    D, rows = population(torch)
    launches = []

    class Lib:
        def einspline_gb300_det_update_accepted_mark(self, *a):
            launches.append(a)
            return 0

    monkeypatch.setattr(api, "_lib", Lib)
    monkeypatch.setattr(api, "_stream", lambda torch, stream: 5)
    as_given = lambda v: v if make == "list" else torch.tensor(v, dtype=getattr(torch, make))  # noqa: E731
    with pytest.raises(IndexError):
        D.update(1, as_given([0, bad, 1]), rows)
    with pytest.raises(IndexError):
        D.update(1, as_given([0, 2]), rows[:2])  # beyond the rows
    assert not launches
    D.update(1, as_given([0, -3, 2]), rows)
    assert len(launches) == 1


def test_status_words_change_owners(monkeypatch):
    """What the GPU may still write for a word's former owner is not read as
    the new owner's, and does not hide the new owner's own refusal."""
    import copy
    import ctypes
    torch = pytest.importorskip("torch")
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda t: t)
    monkeypatch.setattr(api._StatusWord, "_free", type(api._StatusWord._free)())

    def refuse(address, mark):  # the kernel's atomicMax
        w = ctypes.c_int.from_address(address)
        w.value = max(w.value, mark)

    words = [api._StatusWord() for _ in range(70)]
    assert len({w.address for w in words}) == 70
    address, mark = words[5].address, words[5].mark
    words[5] = None
    new = api._StatusWord()
    assert new.address == address and new.mark > mark
    refuse(address, mark)
    assert not new.refused()
    refuse(address, new.mark)
    refuse(address, mark)
    assert new.refused() and not new.refused()
    refuse(address, new.mark)
    other = copy.deepcopy(new)
    assert other.address != address and not other.refused() and new.refused()


def test_no_rows_are_needed_without_an_accepted_walker():
    torch = pytest.importorskip("torch")
    D, _ = population(torch)
    assert D.update(1, [], None) is None
    assert D.update(1, torch.zeros(0, dtype=torch.int64), None) is None
