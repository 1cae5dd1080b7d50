"""When the clearance field stands: the counts by which other tests compare checks with it and without
it do bring it about and do not, for every kind of object, and a change of the environment ends it."""
import pytest

from test_gpu_field import SCENES, WITH, WITHOUT, _base, _configurations

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene", SCENES, ids=lambda f: f.__name__[1:])
def test_the_counts_of_the_field_tests(scene):
    import torch

    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    rb = vg.panda
    q = torch.from_numpy(_configurations(rb, WITH, 21)).cuda()
    env = scene()
    assert not env.field_ready()
    rb.validate_batch(q[:WITHOUT], env)
    assert not env.field_ready()
    env = scene()
    rb.validate_batch(q, env)
    assert env.field_ready()
    env.add_sphere([3.0, 3.0, 3.0, 0.1])
    assert not env.field_ready()
    rb.validate_batch(q[:WITHOUT], env)
    assert not env.field_ready()
    rb.validate_batch(q[:WITH - WITHOUT], env)
    assert env.field_ready()
    # motions count as 64 configurations each
    a, b = (torch.from_numpy(x).cuda() for x in scenes.edges(rb.s_m, rb.s_a, 2500, 6))
    for n, stands in ((2000, False), (2500, True)):
        env = scene()
        rb.validate_motion_batch(a[:n], b[:n], env)
        assert env.field_ready() is stands
    blocks = q[:8 * 12_000].reshape(-1, 8, rb.dimension())
    env = scene()
    rb.fkcc_blocks(blocks, env)
    assert not env.field_ready()


def test_a_stream_under_capture_does_not_build_it():
    import torch

    import vamp_gb300 as vg

    env = _base()
    q = torch.from_numpy(_configurations(vg.panda, WITH, 24)).cuda()
    vg.panda.validate_batch(q[:1000], env)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        vg.panda.validate_batch(q, env)
    assert not env.field_ready()
    vg.panda.validate_batch(q[:1000], env)
    assert env.field_ready()
