"""The coefficient solve of 3D FP32 tables (solve_line.cu: factored
recurrences in FP64, rounded once) against the oracle's FP64 elimination:
axis lengths at the edges of its tiles and where the other solve takes over,
batch widths around its column tiles, and data whose conversions take the
rare forms."""
import numpy as np
import pytest

from einspline_gb300 import api, synth

from helpers import build_pair

P, D1, D2, FL, NA, AP = 0, 1, 2, 3, 4, 5

# Both solves compute in FP64 and round once: half a unit in the last place
# of FP32 (2^-24 relative, at most 2^-150 absolute for subnormal results)
# plus FP64 rounding errors carried along three axes, bounded by 64 units of
# the largest coefficient.
EPS32, EPS64 = 2.0 ** -24, 64 * 2.0 ** -53


def check(orc, kind, grids, bcs, N, data=None, seed=5):
    G, T, _ = build_pair(orc, kind, grids, bcs, N, seed=seed, data=data)
    t, _ = G.table_host()
    got = t[..., :N * G.ncomp].astype(np.float64).reshape(T.coefs64.shape)
    ref = T.coefs64
    scale = np.abs(ref).max()
    bound = np.abs(ref) * EPS32 * (1 + 2.0 ** -20) + scale * EPS64 + 2.0 ** -150
    bad = np.abs(got - ref) > bound
    assert not bad.any(), (np.argwhere(bad)[0], got[bad][0], ref[bad][0])


@pytest.mark.gpu
@pytest.mark.parametrize("axis", range(3))
@pytest.mark.parametrize("M", [4, 5, 7, 8, 9, 15, 17, 63, 64, 72, 73, 144, 145, 288, 289])
def test_axis_lengths(orc, axis, M):
    grids = [(0.0, 1.0, 6)] * 3
    grids[axis] = (0.0, 1.0, M)
    for bc in ((P, P), (AP, AP), (NA, FL), (D1, D2, 0.7, 0.0, -1.3, 0.0)):
        bcs = [(P, P), (D2, NA, 0.2, 0.0, 0.0, 0.0), (AP, AP)]
        bcs[axis] = bc
        check(orc, "s", grids, bcs, 3, seed=M)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", "sc")
@pytest.mark.parametrize("N", [1, 2, 3, 4, 7, 8, 9, 16, 33])
def test_batch_widths(orc, kind, N):
    check(orc, kind, [(0.0, 1.0, 7), (0.0, 2.0, 5), (0.0, 1.0, 9)], [(P, P), (FL, NA), (AP, AP)], N, seed=N)


@pytest.mark.gpu
def test_extreme_data(orc):
    """Zeros, subnormals and magnitudes from 2^-140 to 2^120 in one table."""
    M, N = (12, 11, 10), 6
    rng = np.random.default_rng(3)
    data = np.ldexp(synth.grid_data_uniform(4, M, N, np.float64), rng.integers(-140, 120, size=(N,) + M)).astype(np.float32)
    data[1] = 0.0
    data[2] = np.ldexp(data[2].astype(np.float64) / np.abs(data[2]).max(), -135).astype(np.float32)
    data[3].reshape(-1)[::7] = -0.0
    grids = [(0.0, 1.0, m) for m in M]
    for s in range(N):  # one spline at a time: the bound is relative to its own largest coefficient
        check(orc, "s", grids, [(P, P), (NA, NA), (AP, AP)], 1, data=data[s:s + 1])
