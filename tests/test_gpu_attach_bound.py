"""The extended same-edge check's containing sphere of an attachment: verdicts and block counts are the
oracle's for transforms that turn, scale and skew, no spheres, one, and the most, and radii of zero,
negative and infinite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cases():
    rng = np.random.default_rng(12)
    turn = np.eye(4, dtype=np.float32)
    turn[:3, :3] = [[0.36, 0.48, -0.8], [-0.8, 0.6, 0.0], [0.48, 0.64, 0.6]]
    turn[:3, 3] = [0.05, -0.02, 0.15]
    scale = turn.copy()
    scale[:3, :3] *= 1.7
    skew = np.eye(4, dtype=np.float32)
    skew[0, 1], skew[2, 0], skew[2, 3] = 0.9, -0.4, 0.1
    many = np.concatenate([rng.uniform(-0.15, 0.15, (64, 3)), rng.uniform(0.005, 0.03, (64, 1))], axis=1)
    yield "none", turn, np.zeros((0, 4))
    yield "one", turn, np.array([[0.02, 0.01, 0.05, 0.06]])
    yield "most", turn, many
    yield "scaled", scale, many[:20]
    yield "skewed", skew, many[:9]
    yield "radii", turn, np.array([[0, 0, 0.1, 0.0], [0.1, 0, 0, -0.04], [0, 0.1, 0, 0.03]])
    yield "infinite", turn, np.array([[0, 0, 0.1, 0.02], [0, 0, 0, np.inf]])


@pytest.mark.parametrize("lanes", [8, 4])
@pytest.mark.parametrize("robot", ["panda", "ur5", "fetch", "baxter"])
@pytest.mark.parametrize("name,tf,spheres", list(_cases()), ids=[c[0] for c in _cases()])
def test_edges_with_an_attachment(port, name, tf, spheres, robot, lanes):
    import torch

    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    rb, pr = getattr(vg, robot), port.robot(robot)
    mode = vg.SQRT_X86 if lanes == 8 else vg.SQRT_EXACT
    scene = {**scenes.scene_config1(3), "attachment": {"tf": tf, "spheres": spheres.astype(np.float32)}}
    env, penv = vg.Environment.from_scene(scene, lanes, mode), port.env(scene, mode)
    a, b = scenes.edges(rb.s_m, rb.s_a, 60, 17)
    b = (a + 0.2 * (b - a)).astype(np.float32)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    want, count = penv.validate_motions(pr, a, b, rb.resolution(), lanes, threads=8)
    for field in (False, True):
        if field:
            rb.validate_batch(torch.from_numpy(scenes.configurations(rb.s_m, rb.s_a, 140_000, 4)).cuda(), env)
        blocks = torch.empty(len(a), dtype=torch.int32, device="cuda")
        ok = rb.validate_motion_batch(da, db, env, blocks=blocks)
        assert np.array_equal(ok.cpu().numpy(), want)
        assert np.array_equal(blocks.cpu().numpy(), count)
