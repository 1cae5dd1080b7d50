"""The clearance field's cells lie in tiles of 4 x 4 x 2: small spheres scattered over the whole grid, one per
sector and more, so that a cell read from another's place would rule a touching sphere out.
Verdicts with the field equal those without it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cloud", [False, True])
@pytest.mark.parametrize("robot", ["panda", "ur5"])
def test_field_cells_are_found_where_they_were_written(port, robot, cloud):
    import torch

    assert torch.cuda.is_available()
    import vamp_gb300 as vg

    rb, prb = getattr(vg, robot), port.robot(robot)
    rng = np.random.default_rng(150)
    pts = rng.uniform((-1.6, -1.6, -1.0), (1.6, 1.6, 2.2), (2600, 3)).astype(np.float32)
    env = vg.Environment()
    pts = pts[np.linalg.norm(pts - np.array([0.0, 0.0, 0.4], np.float32), axis=1) > 0.5][:1200]
    if cloud:
        env.add_pointcloud(pts, *rb.min_max_radii(), 0.005)
    else:
        for x, y, z in pts:
            env.add_sphere([float(x), float(y), float(z), 0.01])
    q = torch.from_numpy((prb.s_a + prb.s_m * rng.random((262144, prb.dim))).astype(np.float32)).cuda()
    # fewer than the field asks for, so these run every exact query
    before = rb.validate_batch(q[:100000], env)
    with_field = rb.validate_batch(q, env)
    assert torch.equal(with_field[:100000], before)
    assert 0 < int(before.sum()) < len(before)
