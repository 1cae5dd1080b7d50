"""Replays of a batch count towards its environments' clearance fields as other checks do: a batch too
small to bring one about at once has it after as many launches as the threshold asks for, and its
verdicts and block counts stay what they were."""
import pytest

pytestmark = pytest.mark.gpu


def test_replays_bring_the_field_about():
    import torch

    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    robots = (vg.panda, vg.baxter)
    sizes = (512, 300)  # 64 configurations a motion: 4 launches make 131,072, and 7
    envs = [vg.Environment.from_scene(scenes.scene_config1(3 + k)) for k in range(2)]
    batch, outs, want = vg.Batch(), [], []
    for rb, n, env in zip(robots, sizes, envs):
        a, b = (torch.from_numpy(x).cuda() for x in scenes.edges(rb.s_m, rb.s_a, n, 6))
        out, blocks = torch.empty(n, dtype=torch.uint8, device="cuda"), torch.empty(n, dtype=torch.int32, device="cuda")
        batch.add(rb, env, a, b, out, blocks=blocks)
        outs.append((out, blocks))
        fresh, count = vg.Environment.from_scene(scenes.scene_config1(3 + len(want))), torch.empty_like(blocks)
        want.append((rb.validate_motion_batch(a, b, fresh, blocks=count), count))
        assert not fresh.field_ready()
    for launch in range(1, 9):
        for out, blocks in outs:
            out.fill_(7)
            blocks.zero_()
        batch.launch()
        torch.cuda.synchronize()
        for (out, blocks), (ok, count) in zip(outs, want):
            assert torch.equal(out, ok) and torch.equal(blocks, count), launch
        assert [env.field_ready() for env in envs] == [launch >= 4, launch >= 7], launch
