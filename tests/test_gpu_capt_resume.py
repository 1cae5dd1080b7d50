"""Trees whose lists run out of room at one level after another: the build goes on from the level that
did, in trees of one subtree, of several and of several tiles, and the layout stays the host build's."""
import numpy as np
import pytest

from test_gpu_capt_levels import _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,r_max", [(1025, 1e3), (1500, 5.0), (2049, 0.9), (4097, 0.7), (6000, 1.0), (12000, 0.35), (17000, 0.25)])
def test_the_build_goes_on_where_the_room_ran_out(n, r_max):
    rng = np.random.default_rng(n)
    pts = rng.uniform(-0.5, 0.5, (n, 3)).astype(np.float32)
    _same(pts, 0.01, r_max)  # the larger trees take blocks beyond what the pool keeps
    if n <= 4097:
        pts[::3] = np.round(pts[::3] * 8) / 8  # ties and repeats
        _same(pts, 0.0, r_max)
