"""Environments near the limit of a thread block's shared memory (227 KB of records): they are accepted
for every robot, with the records that do not fit beside the robot's own stage read from global memory.
Verdicts and block counts are the oracle's, with the division in a list of cuboids, in one of capsules
and behind a cloud, heightfield and held object, with and without the clearance field."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
THREADS = max(1, min(16, os.cpu_count() or 1))
LIMIT = 227 * 1024


def _around(rng, n):
    """Points in a part of the robots' reach to the side."""
    turn, far = rng.uniform(1.6, 2.6, n), rng.uniform(0.6, 1.2, n)
    return np.stack([far * np.cos(turn), far * np.sin(turn), rng.uniform(0.1, 1.2, n)], axis=1)


def _cuboids(rng, n):
    from vamp_gb300 import scenes

    return np.stack([scenes.cuboid_fields(p, scenes.random_rotation(rng), rng.uniform(0.004, 0.02, 3)) for p in _around(rng, n)])


def _capsules(rng, n):
    from vamp_gb300 import scenes

    p = _around(rng, n)
    return np.stack([scenes.capsule_fields(a, a + rng.uniform(-0.04, 0.04, 3), 0.01) for a in p])


def _spheres(rng, n):
    return np.concatenate([_around(rng, n), rng.uniform(0.004, 0.015, (n, 1))], axis=1).astype(np.float32)


def _scene(kind):
    from vamp_gb300 import scenes

    rng = np.random.default_rng(31)
    if kind == "cuboids":
        return {"cuboids": _cuboids(rng, 3600)}
    if kind == "capsules":
        return {"spheres": _spheres(rng, 4900), "capsules": _capsules(rng, 1500)}
    tf = np.eye(4, dtype=np.float32)
    tf[2, 3] = 0.1
    return {
        "spheres": _spheres(rng, 6800),
        "cuboids": _cuboids(rng, 80),
        "pointclouds": [{"points": _around(rng, 400).astype(np.float32), "r_min": 0.01, "r_max": 0.25, "r_point": 0.004}],
        "heightfields": [scenes.heightfield(5, centre=(0.2, 0.0, -0.3))],
        "attachment": {"tf": tf, "spheres": np.array([[0, 0, 0, 0.03], [0, 0, 0.08, 0.03]], np.float32)},
    }


@pytest.mark.parametrize("kind", ["cuboids", "capsules", "all"])
@pytest.mark.parametrize("robot", ["panda", "ur5", "fetch", "baxter"])
def test_an_environment_of_nearly_the_limit(port, robot, kind):
    import torch

    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    rb, prb = getattr(vg, robot), port.robot(robot)
    scene = _scene(kind)
    env, penv = vg.Environment.from_scene(scene), port.env(scene)
    q = scenes.configurations(rb.s_m, rb.s_a, 1000, 23)
    a, b = scenes.edges(rb.s_m, rb.s_a, 120, 29)
    b = (a + 0.15 * (b - a)).astype(np.float32)
    states = penv.validate_states(prb, q, threads=THREADS)
    want, count = penv.validate_motions(prb, a, b, rb.resolution(), 8, threads=THREADS)
    dq, da, db = (torch.from_numpy(v).cuda() for v in (q, a, b))
    for field in (False, True):
        if field:
            rb.validate_batch(torch.from_numpy(scenes.configurations(rb.s_m, rb.s_a, 140_000, 4)).cuda(), env)
        assert np.array_equal(rb.validate_batch(dq, env).cpu().numpy(), states)
        for schedule in (-1, 0, 2, 3):
            env.set_schedule(schedule)
            blocks = torch.empty(len(a), dtype=torch.int32, device="cuda")
            assert np.array_equal(rb.validate_motion_batch(da, db, env, blocks=blocks).cpu().numpy(), want), schedule
            assert np.array_equal(blocks.cpu().numpy(), count), schedule
        env.set_schedule(-1)
        assert np.array_equal(rb.validate_motion_batch(a[:40], b[:40], env), want[:40])  # host memory
        alike = dq[:200].repeat_interleave(8, 0).reshape(200, 8, -1).contiguous()
        assert np.array_equal(rb.fkcc_blocks(alike, env).cpu().numpy(), states[:200])
    if kind != "all":
        assert 0 < int(states.sum()) < len(q)


@pytest.mark.parametrize("robot", ["panda", "ur5", "fetch", "baxter"])
def test_the_limit_is_the_same_for_every_robot(robot):
    import torch

    import vamp_gb300 as vg
    from vamp_gb300 import scenes
    from vamp_gb300._lib import lib

    rb = getattr(vg, robot)
    q = torch.from_numpy(scenes.configurations(rb.s_m, rb.s_a, 64, 22)).cuda()
    out = torch.empty(64, dtype=torch.uint8, device="cuda")
    cuboids = _cuboids(np.random.default_rng(2), LIMIT // 64 + 1)
    for n, code in ((LIMIT // 64, 0), (LIMIT // 64 + 1, -5)):
        env = vg.Environment.from_scene({"cuboids": cuboids[:n]})
        s = torch.cuda.current_stream().cuda_stream
        assert lib.vg_validate_states_device(rb.name.encode(), env.handle, q.data_ptr(), 64, out.data_ptr(), s) == code


@pytest.mark.parametrize("robot", ["panda", "ur5", "fetch", "baxter"])
def test_sizes_about_the_ones_that_split_the_records(port, robot):
    """All records staged, three eighths left behind for a second resident block, all staged again,
    and left behind because even one block cannot hold them: verdicts are the oracle's each time."""
    import torch

    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    rb, prb = getattr(vg, robot), port.robot(robot)
    stage = {"panda": 65, "ur5": 52, "fetch": 59, "baxter": 114}[robot] * 128 * 4
    pair = (LIMIT + 1024) // 2 - 1024 - stage
    q = scenes.configurations(rb.s_m, rb.s_a, 400, 23)
    a, b = scenes.edges(rb.s_m, rb.s_a, 60, 29)
    b = (a + 0.15 * (b - a)).astype(np.float32)
    cuboids = _cuboids(np.random.default_rng(37), LIMIT // 64)
    for room in (pair, pair * 8 // 5, LIMIT - stage):
        for n in (room // 64 - 1, room // 64, room // 64 + 1):
            scene = {"cuboids": cuboids[:n]}
            env, penv = vg.Environment.from_scene(scene), port.env(scene)
            got = rb.validate_batch(torch.from_numpy(q).cuda(), env).cpu().numpy()
            assert np.array_equal(got, penv.validate_states(prb, q, threads=THREADS)), n
            want, count = penv.validate_motions(prb, a, b, rb.resolution(), 8, threads=THREADS)
            blocks = torch.empty(len(a), dtype=torch.int32, device="cuda")
            ok = rb.validate_motion_batch(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), env, blocks=blocks)
            assert np.array_equal(ok.cpu().numpy(), want) and np.array_equal(blocks.cpu().numpy(), count), n
