"""Autotuning an odd number of values in all: the points, doubles behind the
outputs in one buffer, have to start on 8 bytes (3001 x 203 floats end 4
bytes off)."""
import numpy as np
import pytest

from einspline_gb300 import api, synth
from helpers import build_pair

GRIDS = [(0.0, 1.0, 6), (0.0, 1.0, 5), (0.0, 1.0, 7)]
BCS = [(api.PERIODIC, api.PERIODIC)] * 3


@pytest.mark.gpu
@pytest.mark.parametrize("storage", [api.STORE_NATIVE, api.STORE_I16])
@pytest.mark.parametrize("npts,N", [(1, 1), (3, 5), (301, 203)])
@pytest.mark.parametrize("vgh", [False, True])
def test_odd_counts(orc, storage, npts, N, vgh):
    torch = pytest.importorskip("torch")
    G, _, _ = build_pair(orc, "s", GRIDS, BCS, N, storage=storage)
    pos = torch.from_numpy(synth.points_uniform(3, npts, (0, 0, 0), (1, 1, 1))).cuda()
    before = G.eval(pos, vgh=vgh)
    G.autotune(npts, vgh=vgh)
    for a, b in zip(before, G.eval(pos, vgh=vgh)):
        assert (a is None and b is None) or np.array_equal(a.cpu().numpy(), b.cpu().numpy())
