"""A held object with a sphere whose centre is not finite, or so far out that squared distances
overflow: it touches nothing, and the object's other spheres are tested as ever, against the robot
and the environment.  One with a radius whose square overflows touches everything."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

INF, NAN, FAR = float("inf"), float("nan"), 3e19
GOOD = [[0.1, 0.0, 0.25, 0.08], [0.05, 0.0, 0.4, 0.05], [0.02, 0.03, 0.55, 0.05]]
ODD = {
    "infinite": [[INF, 0.0, 0.0, 0.02]],
    "nan": [[0.0, NAN, 0.0, 0.02]],
    "far": [[FAR, 0.0, 0.0, 0.02]],
    "both-ways": [[INF, 0.0, 0.0, 0.02], [-INF, 0.0, 0.0, 0.02]],
    "largest": [[3e38, 0.0, 0.0, 0.02], [-3e38, 3e38, 0.0, 0.02]],
    "radius": [[0.0, 0.0, 0.0, 1e30]],
}


@pytest.mark.parametrize("first", [True, False], ids=["first", "last"])
@pytest.mark.parametrize("name", list(ODD))
@pytest.mark.parametrize("robot", ["panda", "ur5", "fetch", "baxter"])
def test_a_sphere_that_is_nowhere(port, robot, name, first):
    import torch

    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    rb, pr = getattr(vg, robot), port.robot(robot)
    tf = np.eye(4, dtype=np.float32)
    tf[:3, 3] = [0.02, -0.01, 0.05]
    spheres = np.array(ODD[name] + GOOD if first else GOOD + ODD[name], np.float32)
    scene = {"spheres": np.array([[0.6, 0.2, 0.5, 0.2]]), "attachment": {"tf": tf, "spheres": spheres}}
    good = {**scene, "attachment": {"tf": tf, "spheres": np.array(GOOD, np.float32)}}
    env = vg.Environment.from_scene(scene)
    q = scenes.configurations(rb.s_m, rb.s_a, 2000, 23)
    want = port.env(good).validate_states(pr, q, threads=8)
    if name == "radius":
        want = np.zeros_like(want)
    for field in (False, True):
        if field:
            rb.validate_batch(torch.from_numpy(scenes.configurations(rb.s_m, rb.s_a, 140_000, 4)).cuda(), env)
        assert np.array_equal(rb.validate_batch(torch.from_numpy(q).cuda(), env).cpu().numpy(), want)
    if name != "radius":
        assert 0 < int(want.sum()) < len(q)
