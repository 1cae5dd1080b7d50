"""The check that makes the clearance field due queues its build and returns: it waits for nothing, ends
no capture in another thread, and checks on other streams, batches included, wait on the GPU."""
import threading
import time

import pytest

from test_gpu_field import WITH, WITHOUT, _base, _cloud_host, _configurations

pytestmark = pytest.mark.gpu
SLEEP = 1_000_000_000  # clock cycles, half a second or more


def _inputs(rb, n=WITH):
    import torch

    return torch.from_numpy(_configurations(rb, n, 21)).cuda()


@pytest.mark.parametrize("scene", [_base, _cloud_host], ids=lambda f: f.__name__[1:])
def test_the_call_returns_while_its_stream_is_busy(scene):
    import torch

    import vamp_gb300 as vg
    from vamp_gb300 import scenes

    rb = vg.panda
    q = _inputs(rb)
    want = rb.validate_batch(q, scene())
    a, b = (torch.from_numpy(x).cuda() for x in scenes.edges(rb.s_m, rb.s_a, 1000, 6))
    env, busy, other = scene(), torch.cuda.Stream(), torch.cuda.Stream()
    motions = rb.validate_motion_batch(a, b, env)
    small = rb.validate_batch(q[:1000], env)
    out, out2 = torch.empty_like(want), torch.empty_like(want)
    batch, out3 = vg.Batch(), torch.empty_like(motions)
    batch.add(rb, env, a, b, out3)
    torch.cuda.synchronize()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(SLEEP)
        t0 = time.perf_counter()
        rb.validate_batch(q, env, out=out)
        took = time.perf_counter() - t0
    assert env.field_ready() and not busy.query() and took < 0.1
    with torch.cuda.stream(other):  # these queue behind the build, whose stream is still busy
        rb.validate_batch(q, env, out=out2)
        batch.launch()
    assert not busy.query()
    torch.cuda.synchronize()
    assert torch.equal(out, want) and torch.equal(out2, want) and torch.equal(out3, motions)
    assert torch.equal(small, want[:1000])


def test_another_threads_capture_goes_on():
    import torch

    import vamp_gb300 as vg

    rb = vg.panda
    q = _inputs(rb)
    env, want = _base(), rb.validate_batch(q, _base())
    rb.validate_batch(q[:1000], env)
    out, side = torch.empty_like(want), torch.cuda.Stream()
    x = torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()

    def check():
        with torch.cuda.stream(side):
            rb.validate_batch(q, env, out=out)

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):  # the default mode: unsafe calls of any thread end the capture
        x += 1
        t = threading.Thread(target=check)
        t.start()
        t.join()
        x += 1
    graph.replay()
    torch.cuda.synchronize()
    assert env.field_ready() and bool((x == 2).all()) and torch.equal(out, want)


def test_a_graph_captured_while_the_build_is_queued():
    import torch

    import vamp_gb300 as vg

    rb = vg.panda
    q = _inputs(rb)
    env, want = _base(), rb.validate_batch(q, _base())
    rb.validate_batch(q[:WITHOUT], env)
    busy, out = torch.cuda.Stream(), torch.empty_like(want)
    torch.cuda.synchronize()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(SLEEP)
        rb.validate_batch(q[:WITH - WITHOUT], env)
    assert env.field_ready()
    # torch.cuda.graph would wait for the device first
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(stream):
        graph.capture_begin()
        rb.validate_batch(q, env, out=out)
        graph.capture_end()
        assert not busy.query()
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
