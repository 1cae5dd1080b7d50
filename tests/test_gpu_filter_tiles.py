"""The pointcloud filter at sizes about its sort tile (8192 keys, 256 the smallest), its chunks (1024
entries, 32 of them walked directly) and its tile offsets (2048 tiles added up directly): the kept
points are the oracle's, in order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 255, 256, 257, 1023, 1025, 8191, 8192, 8193, 16384, 16385, 32767, 32769, 65536, 70001])
def test_kept_points(port, n):
    import torch

    import vamp_gb300 as vg

    rng = np.random.default_rng(n)
    pts = rng.uniform(-1, 1, (n, 3)).astype(np.float32)
    pts[::5] = pts[0]  # repeats
    pts[1::7] = np.round(pts[1::7], 1)
    o = np.zeros(3, np.float32)
    for dist, cull in ((0.03, True), (0.0005, False)):
        got = vg.filter_pointcloud_device(torch.from_numpy(pts).cuda(), dist, 1.2, o, o - 0.8, o + 0.9, cull).cpu().numpy()
        want = port.filter_pointcloud(pts, dist, 1.2, o, o - 0.8, o + 0.9, cull)
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


def test_more_tiles_than_are_added_up_directly(port):
    import torch

    import vamp_gb300 as vg

    n = 2048 * 1024 + 4097
    pts = np.random.default_rng(3).uniform(-1, 1, (n, 3)).astype(np.float32)
    o = np.zeros(3, np.float32)
    got = vg.filter_pointcloud_device(torch.from_numpy(pts).cuda(), 0.02, 0.9, o, o - 1, o + 1, True).cpu().numpy()
    assert np.array_equal(got, port.filter_pointcloud(pts, 0.02, 0.9, o, o - 1, o + 1, True))
