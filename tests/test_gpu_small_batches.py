"""Batches too small to fill the GPU run in smaller blocks (fit_tile): the
same bits as the same points in a batch that fills it, and threads launching
one kernel with different block sizes at once do not disturb each other."""
import threading

import pytest

from einspline_gb300 import api

GRID = [(0.0, 1.0, 13), (0.0, 1.0, 9), (0.0, 1.0, 11)]
PER = [(api.PERIODIC, api.PERIODIC)] * 3
SIZES = (1, 2, 3, 5, 8, 9, 31, 48, 130, 300, 1001)


def build(torch, kind, storage, N):
    G = api.MultiUBspline3D(kind, GRID, PER, N, storage=storage)
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    shape = (N,) + G.M + ((2,) if kind in "cz" else ())
    G.set_device(0, torch.rand(shape, generator=g, device="cuda",
                               dtype=torch.float32 if kind in "sc" else torch.float64) - 0.5)
    G.flush()
    g.manual_seed(7)
    return G, torch.rand((6000, 3), generator=g, device="cuda", dtype=torch.float64)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,storage,N", [("s", 0, 1), ("s", 0, 203), ("s", 0, 1030), ("s", api.STORE_F16, 300),
                                            ("s", api.STORE_BF16, 33), ("s", api.STORE_I16, 515), ("c", 0, 65),
                                            ("c", api.STORE_F16, 130), ("d", 0, 130), ("z", 0, 30)])
def test_small_batches_are_bit_identical(kind, storage, N):
    torch = pytest.importorskip("torch")
    G, pos = build(torch, kind, storage, N)
    for vgh in (True, False):
        for sort in (False, True):
            ref = G.eval(pos, vgh=vgh)
            p0 = 0
            for n in SIZES:
                got = G.eval(pos[p0:p0 + n], vgh=vgh, sort=sort)
                for a, b in zip(got, ref):
                    if b is not None:
                        assert torch.equal(a, b[p0:p0 + n]), (vgh, sort, n)
                p0 += n


@pytest.mark.gpu
@pytest.mark.parametrize("storage", [0, api.STORE_F16])
def test_threads_with_different_batch_sizes(storage):
    torch = pytest.importorskip("torch")
    G, pos = build(torch, "s", storage, 300)
    ref = G.eval(pos)
    torch.cuda.synchronize()
    errors = []

    def work(n):
        try:
            s = torch.cuda.Stream()
            for i in range(60):
                with torch.cuda.stream(s):
                    got = G.eval(pos[i:i + n], stream=s)
                s.synchronize()
                if not all(torch.equal(a, b[i:i + n]) for a, b in zip(got, ref)):
                    errors.append((n, i))
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(repr(e))
    ts = [threading.Thread(target=work, args=(n,)) for n in (1, 40, 500, 900, 1500, 5000)]
    for t in ts:
        t.start()
    for t in ts:
        t.join(timeout=120)
    assert not errors, errors[:3]
