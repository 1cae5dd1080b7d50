"""An environment changed while checks on it are queued behind other work, on a stream that does not
synchronise with the default one: they see it as it was when they were called, later ones as it is
now.  The image grows in place, grows out of its room, and shrinks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SLEEP = 200_000_000  # clock cycles, about a tenth of a second


def _case(kind, rb, env, q, goals):
    import vamp_gb300 as vg

    if kind == "states":
        return lambda: rb.validate_batch(q, env)
    if kind == "motions":
        return lambda: rb.validate_motion_batch(q[: len(goals)], goals, env)
    import torch

    batch, out = vg.Batch(), torch.empty(len(goals), dtype=torch.uint8, device="cuda")
    batch.add(rb, env, q[: len(goals)], goals, out)

    def run():
        batch.launch()
        return out.clone()

    return run


@pytest.mark.parametrize("kind", ["states", "motions", "batch"])
def test_queued_checks_see_the_environment_of_their_call(kind):
    import torch

    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    rb = vg.panda
    scene = scenes.scene_config1(3)
    q = torch.from_numpy(scenes.configurations(rb.s_m, rb.s_a, 20_000, 3)).cuda()
    goals = (q[:2000] + 0.1).contiguous()
    extra = [[0.7 * np.cos(1.6 * k + 0.5), 0.7 * np.sin(1.6 * k + 0.5), 0.5, 0.2] for k in range(4)]
    held = vg.Attachment(np.eye(4, dtype=np.float32))
    held.add_spheres([[0, 0, 0.3, 0.3]] * 40)
    # one sphere at a time within the room, then many at once past it, then an object held and let go
    steps = [lambda env, i=i: env.add_sphere(extra[i]) for i in range(3)]
    steps += [lambda env: [env.add_sphere([2.0 + 0.01 * k, 2.0, 0.5, 0.1]) for k in range(200)] + [env.add_sphere(extra[3])]]
    steps += [lambda env: env.attach(held), lambda env: env.detach()]
    # what each state of the environment gives
    want, env = [], vg.Environment.from_scene(scene)
    for step in [None, *steps]:
        if step:
            step(env)
        want.append(_case(kind, rb, env, q, goals)().cpu())
    assert all(not torch.equal(a, b) for a, b in zip(want[:4], want[1:4])) and not torch.equal(want[4], want[5])

    env = vg.Environment.from_scene(scene)
    stream = torch.cuda.Stream()
    check = _case(kind, rb, env, q, goals)
    check()
    torch.cuda.synchronize()
    got = []
    with torch.cuda.stream(stream):
        for step in [None, *steps]:
            if step:
                step(env)
            torch.cuda._sleep(SLEEP)
            got.append(check())
    stream.synchronize()
    for i, (g, w) in enumerate(zip(got, want)):
        assert torch.equal(g.cpu(), w), i
