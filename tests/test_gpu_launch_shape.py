"""The reported launch shape is a large batch's, not a single point's: FP32
vgh on a table that L2 holds runs by direct loads, 32 x 2 threads with 4
points a lane (32 x 4 in cell order)."""
import pytest

from einspline_gb300 import api


@pytest.mark.gpu
@pytest.mark.parametrize("N", [1, 64, 300])
def test_default_shape_of_an_l2_resident_table(N):
    pytest.importorskip("torch")
    G = api.MultiUBspline3D("s", [(0.0, 1.0, 12)] * 3, [(api.PERIODIC, api.PERIODIC)] * 3, N)
    assert G.get_load_mode() == 0
    assert G.get_tile() == (32, 2, 8)
    assert G.launch_shape() == (32, 2, 8, 0)
    assert G.launch_shape(sorted=True) == (32, 4, 16, 0)
