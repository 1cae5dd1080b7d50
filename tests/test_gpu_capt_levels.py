"""The device tree build's tiles and list room: the layout is the host build's at sizes about the
sort tile (one subtree, one full tile, the first levels above it), with ties and repeated points,
and for sphere radii whose lists outgrow the first room and make the build start again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(points, r_min, r_max, r_point=0.0025):
    import torch

    import vamp_gb300 as vg

    host, dev = vg.Environment(), vg.Environment()
    host.add_pointcloud(points, r_min, r_max, r_point)
    dev.add_pointcloud_device(torch.from_numpy(points).cuda(), r_min, r_max, r_point)
    a, b = host.pointcloud_layout(0), dev.pointcloud_layout(0)
    for k in ("tests", "aabbs", "aff_starts", "aff", "top"):
        assert a[k].shape == b[k].shape and np.array_equal(a[k].view(np.uint32), b[k].view(np.uint32)), k


@pytest.mark.parametrize("n", [2, 3, 4, 5, 31, 33, 64, 65, 127, 1024, 1025, 2047, 2048, 2049, 4096, 4097, 9000])
def test_sizes_about_the_tile(n):
    rng = np.random.default_rng(n)
    _same(rng.uniform(-1, 1, (n, 3)).astype(np.float32), 0.01, 0.15)
    _same((rng.integers(0, 5, (n, 3)) * 0.25 - 0.5).astype(np.float32), 0.0, 0.1)  # ties, repeats, -0.0 and 0.0


@pytest.mark.parametrize("n,r_max", [(3000, 0.6), (9000, 0.5)])
def test_lists_that_outgrow_the_first_room(n, r_max):
    rng = np.random.default_rng(7)
    _same(rng.uniform(-0.5, 0.5, (n, 3)).astype(np.float32), 0.01, r_max)
