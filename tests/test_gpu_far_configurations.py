"""Configurations far outside the joint limits: an angle of thousands of radians and more leaves the
sine and cosine it is given inconsistent (they round the angle differently), so frames are no
rotations any more and what is fixed in one does not keep its distances.  Verdicts and block counts
are the oracle's all the same, for every robot, among primitives, with a cloud and with a held object,
with and without the clearance field."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
THREADS = max(1, min(16, os.cpu_count() or 1))


def _far(rng, s_m, s_a, n):
    """Uniform configurations; in each one joint or every joint 10^1.5 to 10^7.5 from there, half of
    them at least 10^6."""
    dim = len(s_m)
    q = s_a + s_m * rng.random((n, dim))
    size = 10.0 ** rng.uniform(np.where(rng.random((n, 1)) < 0.5, 1.5, 6.0), 7.5, (n, 1)) * rng.choice([-1.0, 1.0], (n, dim))
    which = np.where(rng.random((n, 1)) < 0.5, 1.0, (np.arange(dim) == rng.integers(0, dim, (n, 1))))
    return (q + which * size).astype(np.float32)


def _scene(kind):
    from vamp_gb300 import scenes

    scene = dict(scenes.scene_config1(3))
    if kind == "cloud":
        scene["pointclouds"] = [{"points": scenes.surface_pointcloud(4, 2000), "r_min": 0.012, "r_max": 0.25, "r_point": 0.01}]
    if kind == "held":
        tf = np.eye(4, dtype=np.float32)
        tf[2, 3] = 0.1
        balls = np.random.default_rng(5).uniform(-0.3, 0.3, (12, 4))
        balls[:, 3] = 0.03
        scene["attachment"] = {"tf": tf, "spheres": balls.astype(np.float32)}
    return scene


@pytest.mark.parametrize("field", [False, True], ids=["exact", "field"])
@pytest.mark.parametrize("kind", ["primitives", "cloud", "held"])
@pytest.mark.parametrize("robot", ["panda", "ur5", "fetch", "baxter"])
def test_far_configurations(port, robot, kind, field):
    import torch

    assert torch.cuda.is_available()
    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    rb, prb = getattr(vg, robot), port.robot(robot)
    rng = np.random.default_rng(41)
    scene = _scene(kind)
    env, penv = vg.Environment.from_scene(scene), port.env(scene)
    if field:
        rb.validate_batch(torch.from_numpy(scenes.configurations(rb.s_m, rb.s_a, 140_000, 4)).cuda(), env)
    q = _far(rng, prb.s_m, prb.s_a, 200_000)
    got = rb.validate_batch(torch.from_numpy(q).cuda(), env).cpu().numpy()
    assert np.array_equal(got, penv.validate_states(prb, q, threads=THREADS))
    # motions of a few blocks from there
    a = q[:3000]
    b = (a + rng.uniform(-0.4, 0.4, a.shape)).astype(np.float32)
    near = np.linalg.norm((b - a).astype(np.float64), axis=1) < 4.0
    a, b = a[near], b[near]
    assert len(a) > 1000
    want, count = penv.validate_motions(prb, a, b, rb.resolution(), 8, threads=THREADS)
    blocks = torch.empty(len(a), dtype=torch.int32, device="cuda")
    ok = rb.validate_motion_batch(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), env, blocks=blocks)
    assert np.array_equal(ok.cpu().numpy(), want)
    assert np.array_equal(blocks.cpu().numpy(), count)
    if kind == "primitives":
        assert 0 < int(got.sum()) < len(q)
