"""Self checks of single configurations: within a warp only the lanes inside a check's danger box
and not yet found colliding ask for its rows, two rows a step.  An empty environment leaves the
self checks alone; configurations inside the joint limits, at their edges and outside (where every
pair is tested), in full warps, remainders and alone.  Verdicts are the oracle's."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
THREADS = max(1, min(16, os.cpu_count() or 1))


@pytest.mark.parametrize("robot", ["panda", "ur5", "fetch", "baxter"])
@pytest.mark.parametrize("where", ["inside", "edges", "outside", "mixed"])
def test_self_checks_of_configurations(port, robot, where):
    import torch

    assert torch.cuda.is_available()
    import vamp_gb300 as vg

    rb, prb = getattr(vg, robot), port.robot(robot)
    rng = np.random.default_rng(130)
    n = 4097
    u = rng.random((n, prb.dim))
    if where == "edges":
        u = np.where(rng.random(u.shape) < 0.5, np.round(u), u)
    elif where == "outside":
        u = u * 1.6 - 0.3
    elif where == "mixed":
        u[rng.random(n) < 0.02] *= 1.5
    q = (prb.s_a + prb.s_m * u).astype(np.float32)
    env, penv = vg.Environment(), port.env({})
    want = penv.validate_states(prb, q, threads=THREADS)
    dev = torch.from_numpy(q).cuda()
    for m in (1, 31, 33, n):
        assert np.array_equal(rb.validate_batch(dev[:m], env).cpu().numpy(), want[:m]), m
        assert np.array_equal(rb.validate_batch(q[n - m:], env), want[n - m:]), m
    assert 0 < int(want.sum()) < n
