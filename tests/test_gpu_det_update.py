"""The fused inverse update (k_det_update) against float64 algebra: sizes
around its units of four columns, its cluster and block shapes and the
two-pass kernels beyond them, rows and matrices that are not 16-byte
aligned, padding, and more walkers than clusters are resident."""
import numpy as np
import pytest

from einspline_gb300 import api

U = 2.0 ** -24


def run_case(torch, n, ld, trans, W, shift=0, seed=1):
    """shift: floats by which every inverse is offset from 16-byte alignment."""
    rng = np.random.default_rng(seed)
    A = np.zeros((W, ld, ld), np.float32)
    B = np.full((W, ld, ld), np.nan, np.float32)  # padding must neither count nor change
    base = np.eye(n) + 0.3 * rng.standard_normal((n, n)) / np.sqrt(n)
    inv = np.linalg.inv(base)
    s = rng.uniform(0.5, 2.0, (W, n))
    k = (2 * n) // 3
    rows = np.zeros((W, n), np.float32)
    for w in range(W):
        A[w, :n, :n] = s[w][:, None] * base
        m = inv / s[w][None, :]
        B[w, :n, :n] = m.T if trans else m
        rows[w] = A[w, k, :n] + 0.2 / np.sqrt(n) * s[w, k] * rng.standard_normal(n)
    flat = torch.full((W * ld * ld + shift,), float("nan"), device="cuda")
    dB = flat[shift:].view(W, ld, ld)
    dB.copy_(torch.from_numpy(B))
    dA = torch.from_numpy(A).cuda()
    D = api.Determinants(dA, dB, n, trans)
    D.update(k, list(range(W)), torch.from_numpy(rows).cuda())
    torch.cuda.synchronize()
    A2, B2 = dA.cpu().numpy(), dB.cpu().numpy()
    for w in range(W):
        expect = A[w].copy()
        expect[k, :n] = rows[w]
        assert np.array_equal(A2[w], expect)
        b0 = B[w, :n, :n].astype(np.float64)
        b0 = b0.T if trans else b0
        got = B2[w, :n, :n].astype(np.float64)
        got = got.T if trans else got
        delta = rows[w].astype(np.float64) - A[w, k, :n]
        x, colk = delta @ b0, b0[:, k]
        p = -1.0 / (1.0 + x[k])
        ref = b0 + np.outer(colk, x) * p
        # FP32 sums of n products in any order: n + 1 units of their magnitudes
        S = (n + 1) * (np.abs(delta) @ np.abs(b0))
        rel_p = abs(p) * S[k] + 3
        bound = 2 * U * (np.abs(ref) + np.abs(colk)[:, None] * abs(p) * (S + np.abs(x) * (rel_p + 3))[None, :])
        assert (np.abs(got - ref) <= bound).all(), (n, ld, trans, w)
        pad = B2[w].copy()
        pad[:n, :n] = np.nan
        assert np.isnan(pad).all()


SIZES = [1, 2, 3, 4, 5, 15, 63, 64, 65, 126, 99, 100, 101, 127, 128, 160, 161, 200, 240, 241, 360, 361, 500, 501, 513]


@pytest.mark.gpu
@pytest.mark.parametrize("trans", [0, 1])
@pytest.mark.parametrize("n", SIZES)
def test_sizes_and_paddings(n, trans):
    torch = pytest.importorskip("torch")
    for ld in (n, n + 1, (n + 7) // 4 * 4):
        run_case(torch, n, ld, trans, 3, seed=n)


@pytest.mark.gpu
@pytest.mark.parametrize("trans", [0, 1])
@pytest.mark.parametrize("n", [2045, 2048, 2049])
def test_largest(n, trans):
    torch = pytest.importorskip("torch")
    run_case(torch, n, (n + 3) // 4 * 4, trans, 1, seed=n)


@pytest.mark.gpu
@pytest.mark.parametrize("trans", [0, 1])
@pytest.mark.parametrize("n", [6, 96, 130, 200, 324, 390, 506])
def test_matrices_off_16_byte_alignment(n, trans):
    torch = pytest.importorskip("torch")
    for shift in (1, 2, 3):
        run_case(torch, n, (n + 3) // 4 * 4, trans, 3, shift=shift, seed=n + shift)


@pytest.mark.gpu
@pytest.mark.parametrize("trans", [0, 1])
@pytest.mark.parametrize("n,W", [(12, 2500), (130, 700), (164, 400), (244, 300), (364, 200), (524, 60)])
def test_more_walkers_than_clusters(n, W, trans):
    torch = pytest.importorskip("torch")
    run_case(torch, n, (n + 3) // 4 * 4, trans, W, seed=n)
