"""A warp takes fewer configurations (or blocks) where a batch is small, by how many warps are resident:
batches about every such step, for robots with different residency, and their verdicts equal the
ones the same configurations get in a batch that fills the warps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("robot", ["panda", "baxter"])
@pytest.mark.parametrize("cloud", [False, True])
def test_small_batches_equal_full_warps(port, robot, cloud):
    import torch

    assert torch.cuda.is_available()
    import vamp_gb300 as vg

    rb, prb = getattr(vg, robot), port.robot(robot)
    rng = np.random.default_rng(140)
    env8, env4 = vg.Environment(), vg.Environment(lanes=4)
    pts = rng.uniform((0.3, -1.0, 0.0), (1.2, 1.0, 1.2), (3000, 3)).astype(np.float32)
    for env in (env8, env4):
        for x, y, z in pts[:40]:
            env.add_sphere([float(x), float(y), float(z), 0.03])
        if cloud:
            env.add_pointcloud(pts[40:], *rb.min_max_radii(), 0.005)
    q = torch.from_numpy((prb.s_a + prb.s_m * rng.random((200000, prb.dim))).astype(np.float32)).cuda()
    want = rb.validate_batch(q, env8)
    assert 0 < int(want.sum()) < len(q)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    sizes = {1, 2, 33}
    for warps in (8, 12, 16, 20, 24):
        sizes |= {sms * warps * share + d for share in (1, 2, 4, 8, 16) for d in (0, 1)}
    for n in sorted(sizes):
        assert torch.equal(rb.validate_batch(q[-n:], env8), want[-n:]), n
    for env, lanes in ((env8, 8), (env4, 4)):
        full = rb.fkcc_blocks(q[: 20000 * lanes].reshape(-1, lanes, prb.dim), env)
        for warps in (1, 12, 16, 20):
            for n in (sms * warps, sms * warps + 1, 2 * sms * warps + 1):
                n = min(n, 20000)
                assert torch.equal(rb.fkcc_blocks(q[: n * lanes].reshape(-1, lanes, prb.dim), env), full[:n]), (lanes, n)
