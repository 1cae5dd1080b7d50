"""Motions checked in a caller's own graph: a replay gives its verdicts and block counts whatever the
environment's other calls needed in scratch since the capture."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [8, 4])
def test_a_captured_check_outlives_larger_batches(lanes):
    import torch

    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    rb = vg.panda
    env = vg.Environment.from_scene(scenes.scene_config1(3), lanes, vg.SQRT_X86 if lanes == 8 else vg.SQRT_EXACT)
    a, b = (torch.from_numpy(v).cuda() for v in scenes.edges(rb.s_m, rb.s_a, 65_536, 17))
    n = 8192  # enough edges for a hand-out order
    want = torch.empty(len(a), dtype=torch.int32, device="cuda")
    ok = rb.validate_motion_batch(a[:n], b[:n], env, blocks=want[:n])  # the usual warm-up
    ins = [a[:n].clone(), b[:n].clone()]
    blocks = torch.zeros(n, dtype=torch.int32, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = rb.validate_motion_batch(*ins, env, blocks=blocks)
    all_ok = rb.validate_motion_batch(a, b, env, blocks=want)  # needs more scratch than the warm-up
    other = torch.zeros(64 << 20, dtype=torch.uint8, device="cuda")  # may take up what was given back
    for at in (0, n, 5 * n):
        ins[0].copy_(a[at:at + n])
        ins[1].copy_(b[at:at + n])
        out.zero_()
        blocks.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, all_ok[at:at + n]) and torch.equal(blocks, want[at:at + n]), at
    assert torch.equal(ok, all_ok[:n]) and not bool(other.any())
