"""The kernel that checks every block of a small host batch of edges at once, against the edge
kernels (which take CUDA tensors): batches that end inside a warp's last segments, that fill up to the
4,096 blocks the path takes, with motion vectors, in both lane widths, with the extended tests and
with an environment so large that the grid is short and a warp takes several rounds.  Verdicts
are equal, byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def vg():
    import torch

    assert torch.cuda.is_available()
    import vamp_gb300 as vg

    return vg


def _env(vg, kind, lanes):
    from vamp_gb300 import scenes

    rng = np.random.default_rng(121)
    if kind == "large":
        env = vg.Environment(lanes=lanes)
        for x, y, z, r in rng.uniform((0.4, 0.4, 0.0, 0.01), (1.9, 1.9, 1.5, 0.05), (2000, 4)):
            env.add_sphere([x, y, z, r])
        return env
    env = vg.Environment.from_scene(scenes.scene_config1(120), lanes=lanes)
    if kind == "heightfield":
        h = rng.uniform(0.0, 0.05, (9, 9)).astype(np.float32)
        env.add_heightfield(vg.make_heightfield((0.0, 0.0, -0.2), (0.25, 0.25, 1.0), (9, 9), h.reshape(-1)))
    return env


@pytest.mark.parametrize("robot,kind", [("panda", "plain"), ("panda", "heightfield"), ("panda", "large"), ("ur5", "plain"),
                                        ("fetch", "heightfield"), ("baxter", "large")])
@pytest.mark.parametrize("lanes", [8, 4])
def test_edge_blocks_equal_the_edge_kernels(vg, robot, kind, lanes):
    import torch

    from vamp_gb300 import scenes

    rb = getattr(vg, robot)
    env, resolution = _env(vg, kind, lanes), rb.resolution()
    a, b = scenes.edges(rb.s_m, rb.s_a, 600, 122)
    b = (a + (b - a) * np.random.default_rng(123).uniform(0.02, 0.4, (len(a), 1))).astype(np.float32)
    v = b - a
    d = np.linalg.norm(v, axis=1).astype(np.float32)
    # blocks as the path counts them, give or take the last ulp: the largest batch just under its limit
    nb = np.maximum(np.ceil(d / np.float32(lanes) * resolution), 1).astype(int)
    most = int(np.searchsorted(np.cumsum(nb), 4096 - 64))
    for n in (1, 2, 5, 17, 129, min(most, len(a))):
        dev = [torch.from_numpy(x[:n]).cuda() for x in (a, b, v, d)]
        want = rb.validate_motion_batch(dev[0], dev[1], env, resolution).cpu().numpy()
        got = rb.validate_motion_batch(a[:n], b[:n], env, resolution)
        assert np.array_equal(got, want), n
        want = rb.validate_vector_batch(dev[0], dev[2], dev[3], env, resolution).cpu().numpy()
        got = rb.validate_vector_batch(a[:n], v[:n], d[:n], env, resolution)
        assert np.array_equal(got, want), n
    assert 0 < int(want.sum()) < len(want)
