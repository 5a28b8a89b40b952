"""The single-point kernel (k_point) against the batched kernels on the same
table, bit for bit: column counts around its blocks of 128 (FP64: 32)
columns, every storage, every output form, points outside the box, and calls
interleaved with batched ones."""
import numpy as np
import pytest

from einspline_gb300 import api

GRID = [(0.0, 1.0, 9), (-1.0, 1.0, 7), (0.5, 2.5, 8)]
BCS = [(api.PERIODIC,) * 2, (api.NATURAL,) * 2, (api.ANTIPERIODIC,) * 2]
POINTS = [(0.1, 0.2, 0.7), (0.999, -0.999, 2.499), (0.0, 1.0, 0.5), (-0.3, 1.4, 2.7)]


@pytest.mark.gpu
@pytest.mark.parametrize("kind,storage", [("s", 0), ("s", api.STORE_F16), ("s", api.STORE_BF16), ("s", api.STORE_I16),
                                          ("c", 0), ("c", api.STORE_F16), ("d", 0), ("z", 0)])
@pytest.mark.parametrize("N", [1, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 300])
def test_point_equals_batch(kind, storage, N):
    torch = pytest.importorskip("torch")
    G = api.MultiUBspline3D(kind, GRID, BCS, N, storage=storage)
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    shape = (N,) + G.M + ((2,) if kind in "cz" else ())
    G.set_device(0, torch.rand(shape, generator=g, device="cuda",
                               dtype=torch.float32 if kind in "sc" else torch.float64) - 0.5)
    G.flush()
    pos = torch.tensor(POINTS, dtype=torch.float64, device="cuda")
    G.set_load_mode(0)  # the FMA kernels, also for F16 and BF16
    v, gr, h = (x.cpu().numpy() for x in G.eval(pos, layout=1))
    G.set_load_mode(-1)
    for i, p in enumerate(POINTS):
        a = G.eval_point(*p)
        assert np.array_equal(a[0], v[i]) and np.array_equal(a[1], gr[i]) and np.array_equal(a[2], h[i])
        assert np.array_equal(G.eval_point(*p, vgh=False)[0], v[i])
        b = G.eval_point_vg(*p)
        assert np.array_equal(b[0], v[i]) and np.array_equal(b[1], gr[i])
        b = G.eval_point_vgl(*p)
        assert np.array_equal(b[0], v[i]) and np.array_equal(b[1], gr[i])
        assert np.array_equal(b[2], (h[i][:, 0, 0] + h[i][:, 1, 1]) + h[i][:, 2, 2])
    G.set_load_mode(1)  # a forced mode takes the batched kernel
    assert np.array_equal(G.eval_point(*POINTS[0])[2], h[0])
