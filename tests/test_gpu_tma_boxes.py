"""Load mode 4 with a number of columns whose rounded block width is not a
whole number of tensor-map boxes: the block narrows to whole boxes (its copies
otherwise brought fewer bytes than the stage waits for)."""
import pytest

from einspline_gb300 import api


@pytest.mark.gpu
@pytest.mark.parametrize("kind,N", [("s", 257), ("s", 384), ("s", 600), ("d", 264), ("d", 330)])
def test_blocks_of_whole_boxes(kind, N):
    torch = pytest.importorskip("torch")
    dt = torch.float32 if kind == "s" else torch.float64
    G = api.MultiUBspline3D(kind, [(0.0, 1.0, 6)] * 3, [(api.PERIODIC, api.PERIODIC)] * 3, N)
    G.set_device(0, torch.rand((N,) + G.M, device="cuda", dtype=dt) - 0.5)
    G.flush()
    if kind == "d":
        G.set_fp64_mode(1)
    pos = torch.rand((100, 3), device="cuda", dtype=torch.float64)
    G.set_load_mode(0)
    ref = G.eval(pos)
    G.set_load_mode(4)
    got = G.eval(pos)
    for a, b in zip(got, ref):
        assert torch.equal(a, b)
