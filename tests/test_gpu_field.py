"""The clearance field: checks that skip exact queries by it give the verdicts and block counts of
checks without it (and the oracle's), for every kind of object and the odd forms they accept.

The field is built once the states checked in an environment since its last change reach a
threshold; WITH is above it in one call and WITHOUT below it, in an environment of its own.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WITH, WITHOUT = 140_000, 130_000
INF = float("inf")


def _base():
    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    return vg.Environment.from_scene(scenes.scene_config1(3))


def _odd_primitives():
    """Skewed and scaled cuboid axes, lists that do not fit their object's shape, wrong rdv, points
    for segments, huge and far objects, and distances that are not the objects' own."""
    env = _base()
    env.add_primitive(3, [0.7, 0.2, 0.5, 2, 0, 0, 0.5, 1, 0, 0, 0.3, 0.6, 0.1, 0.2, 0.05], 0.1)
    env.add_primitive(3, [-0.6, 0.3, 0.7, 0.1, 0, 0, 0, 0.1, 0, 0, 0, 0.1, 0.02, 0.01, 0.01], 0.2)
    env.add_primitive(4, [0.2, -0.8, 0.6, 0.6, 0.8, 0.5, -0.8, 0.6, 0.5, 0, 0, 1, 0.1, 0.1, 0.2], 0.4)
    env.add_primitive(2, [0.1, 0.8, 0.2, 0.4, 0.3, 0.5, 0.05, 4.0], 0.3)
    env.add_primitive(1, [-0.5, -0.6, 0.3, 0.3, 0.1, 0.2, 0.06, 100.0], 0.3)
    env.add_primitive(1, [-0.2, -0.8, 0.9, 0, 0, 0, 0.08, INF], 0.5)
    env.add_primitive(0, [0.0, 0.0, 60.9, 59.5], 0.7)
    env.add_primitive(0, [0.9, 0.5, 0.4, -0.1], 0.6)
    env.add_primitive(0, [0.4, 0.6, 0.9, 0.1], 3.0)
    env.add_primitive(3, [0, 0, -1005.3, 1, 0, 0, 0, 1, 0, 0, 0, 1, 1000, 1000, 1005], 0.2)
    return env


def _not_finite():
    env = _base()
    env.add_primitive(0, [0.5, float("nan"), 0.4, 0.1], 0.4)
    env.add_primitive(3, [0.5, 0.4, 0.6, 1, 0, 0, 0, 1, 0, 0, 0, INF, 0.1, 0.1, 0.1], 0.4)
    return env


def _points(n=3000):
    from vamp_gb300 import scenes

    far = np.array([[1e6, 0, 0], [0, 0, -50.0], [1.9, 0.2, 0.4], [0.3, -1.7, 0.5]], np.float32)
    return np.concatenate([scenes.surface_pointcloud(4, n), far])


def _cloud_host():
    env = _base()
    env.add_pointcloud(_points(), 0.012, 0.25, 0.0025)
    return env


def _cloud_device():
    import torch

    env = _base()
    env.add_pointcloud_device(torch.from_numpy(_points()).cuda(), 0.012, 0.25, 0.03)
    return env


def _cloud_layout():
    """A tree given as a layout whose points are not all its leaves' own."""
    src = _cloud_host().pointcloud_layout(0)
    src["aff"] = src["aff"].copy()
    src["aff"][:, ::3, 0] += 0.05
    env = _base()
    env.add_pointcloud_layout({**src, "radii": (0.012, 0.25, 0.0025)})
    return env


def _terrain():
    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    env = _base()
    h = scenes.heightfield(5, centre=(0.2, 0.0, -0.3))
    env.add_heightfield(vg.HeightField(h["centre"], h["scale"], (h["xd"], h["yd"]), h["data"]))
    rng = np.random.default_rng(8)
    env.add_heightfield(vg.HeightField((0.1, 0.2, -0.2), (0.004, 0.005, -4.0), (300, 200), rng.random(60000)))
    tf = np.eye(4, dtype=np.float32)
    tf[2, 3] = 0.1
    held = vg.Attachment(tf)
    held.add_spheres([[0, 0, 0, 0.05], [0, 0, 0.1, 0.0], [0.05, 0, 0.1, -0.03]])
    env.attach(held)
    return env


SCENES = [_base, _odd_primitives, _not_finite, _cloud_host, _cloud_device, _cloud_layout, _terrain]


def _configurations(rb, n, seed):
    """Uniform configurations, some beyond the joint limits, a few not finite."""
    from vamp_gb300 import scenes

    q = scenes.configurations(rb.s_m, rb.s_a, n, seed)
    q[::7] += np.float32(0.5)
    q[::5003, 0] = np.nan
    q[1::5003, -1] = INF
    return q


@pytest.mark.parametrize("robot", ["panda", "ur5", "fetch", "baxter"])
@pytest.mark.parametrize("scene", SCENES, ids=lambda f: f.__name__[1:])
def test_states_and_blocks_are_those_of_checks_without_the_field(scene, robot):
    import torch

    import vamp_gb300 as vg

    rb = getattr(vg, robot)
    q = torch.from_numpy(_configurations(rb, WITH, 21)).cuda()
    env = scene()
    got = rb.validate_batch(q, env)
    want = rb.validate_batch(q[:WITHOUT], scene())
    assert torch.equal(got[:WITHOUT], want)
    blocks = q[:8 * 12_000].reshape(-1, 8, rb.dimension())
    assert torch.equal(rb.fkcc_blocks(blocks, env), rb.fkcc_blocks(blocks, scene()))


@pytest.mark.parametrize("schedule", [0, 1, 2, 3])
@pytest.mark.parametrize("lanes", [8, 4])
@pytest.mark.parametrize("robot", ["panda", "ur5", "fetch", "baxter"])
@pytest.mark.parametrize("scene", [_odd_primitives, _cloud_device], ids=lambda f: f.__name__[1:])
def test_edges_are_those_of_checks_without_the_field(scene, robot, lanes, schedule):
    import torch

    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    rb = getattr(vg, robot)
    mode = vg.SQRT_X86 if lanes == 8 else vg.SQRT_EXACT
    a, b = (torch.from_numpy(x).cuda() for x in scenes.edges(rb.s_m, rb.s_a, 2500, 6))
    result = []
    for use in (True, False):
        env = scene()
        env.set_mode(lanes, mode)
        env.set_schedule(schedule)
        if use:
            rb.validate_batch(torch.from_numpy(_configurations(rb, WITH, 22)).cuda(), env)
        n = len(a) if use else 2000
        blocks = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        result.append((rb.validate_motion_batch(a[:n], b[:n], env, blocks=blocks)[:2000], blocks[:2000]))
    assert torch.equal(result[0][0], result[1][0])
    assert torch.equal(result[0][1], result[1][1])


@pytest.mark.parametrize("robot", ["panda", "ur5", "fetch", "baxter"])
def test_verdicts_with_the_field_are_the_oracles(port, robot):
    import torch

    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    rb, pr = getattr(vg, robot), port.robot(robot)
    scene = {**scenes.scene_config1(5), "pointclouds": [
        {"points": scenes.surface_pointcloud(5, 2000), "r_min": 0.012, "r_max": 0.25, "r_point": 0.0025}]}
    env, penv = vg.Environment.from_scene(scene), port.env(scene)
    q = scenes.configurations(rb.s_m, rb.s_a, WITH, 9)
    got = rb.validate_batch(torch.from_numpy(q).cuda(), env).cpu().numpy()
    assert np.array_equal(got[:4096], penv.validate_states(pr, q[:4096], threads=8))
    a, b = scenes.edges(rb.s_m, rb.s_a, 200, 10)
    blocks = torch.empty(200, dtype=torch.int32, device="cuda")
    ok = rb.validate_motion_batch(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), env, blocks=blocks)
    want, count = penv.validate_motions(pr, a, b, rb.resolution(), threads=8)
    assert np.array_equal(ok.cpu().numpy(), want) and np.array_equal(blocks.cpu().numpy(), count)


def test_a_change_of_the_environment_drops_the_field():
    import torch

    import vamp_gb300 as vg

    env = _base()
    q = torch.from_numpy(_configurations(vg.panda, WITH, 23)).cuda()
    before = vg.panda.validate_batch(q, env)
    env.add_sphere([0.45, 0.0, 0.6, 0.3])
    fresh = _base()
    fresh.add_sphere([0.45, 0.0, 0.6, 0.3])
    want = vg.panda.validate_batch(q[:WITHOUT], fresh)
    for _ in range(2):  # without the field again, then with the new one
        assert torch.equal(vg.panda.validate_batch(q[:WITHOUT], env), want)
    assert not torch.equal(before[:WITHOUT], want)


def test_a_stream_under_capture_runs_without_building_the_field():
    import torch

    import vamp_gb300 as vg

    env = _base()
    q = torch.from_numpy(_configurations(vg.panda, WITH, 24)).cuda()
    vg.panda.validate_batch(q[:1000], env)  # uploads the environment
    out = torch.zeros(WITH, dtype=torch.uint8, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        vg.panda.validate_batch(q, env, out=out)
    graph.replay()
    want = vg.panda.validate_batch(q, env)
    torch.cuda.synchronize()
    assert torch.equal(out, want)


@pytest.mark.parametrize("n", [6143, 6144, 6145, 7168, 20001])
def test_motions_handed_out_long_ones_first_are_those_handed_out_as_given(n):
    """Edge counts about the threshold and the rank kernel's tiles: verdicts and block counts land on
    their own edges (the segment-per-edge schedule takes edges as given)."""
    import torch

    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    rb = vg.ur5
    a, b = scenes.edges(rb.s_m, rb.s_a, n, 31)
    rng = np.random.default_rng(2)
    b = a + (b - a) * rng.random((n, 1), dtype=np.float32) ** 4  # many one-block edges
    b[::97] = a[::97] + 300.0  # more blocks than the kernel tells apart
    a, b = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    result = []
    for schedule in (1, 0):
        env = _base()
        env.set_schedule(schedule)
        blocks = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        result.append((rb.validate_motion_batch(a, b, env, blocks=blocks), blocks))
    assert torch.equal(result[0][0], result[1][0]) and torch.equal(result[0][1], result[1][1])
