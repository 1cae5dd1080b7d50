"""The training step's two kernels against the CPU oracle at the sizes where they can go wrong: one
row tile and several, a ragged last tile, fewer tiles than the ring has stages and more, every
padded input width (16, 32, 48, 64), and a step of Adam against the gradients it should follow.

Tolerances are those of test_gpu_mlp.py's gradient test: the oracle rounds where the kernels hold
BF16 values, so only FP32 accumulation differs (per parameter block, 2e-3 of its largest gradient
and 1e-3 in the L2 norm)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(n, dim, seed):
    import torch

    rng = np.random.default_rng(seed)
    q = rng.uniform(-3.0, 3.0, (n, dim)).astype(np.float32)
    valid = (rng.random(n) < 0.6).astype(np.uint8)
    return torch.from_numpy(q).cuda(), torch.from_numpy(valid).cuda()


def _gradients(lib, m, q, valid, dim):
    from oracle import mlp

    count = lib.vg_mlp_param_count(dim)
    grads, loss = np.zeros(count, np.float32), np.zeros(1, np.float32)
    feats = np.zeros((len(q), mlp.kin_of(dim)), np.float32)
    assert lib.vg_mlp_gradients(m, q.data_ptr(), valid.data_ptr(), len(q), grads.ctypes.data, loss.ctypes.data,
                                feats.ctypes.data) == 0, lib.vg_last_error()
    return grads, float(loss[0]), feats


@pytest.mark.parametrize("n,dim", [(1, 7), (127, 6), (128, 7), (129, 8), (512, 14), (640, 7), (1000, 16), (300, 20), (257, 32)])
def test_gradients(n, dim):
    from oracle import mlp
    from vamp_gb300._lib import lib

    q, valid = _inputs(n, dim, n + dim)
    m = lib.vg_mlp_create(dim, 3)
    try:
        params = np.zeros(lib.vg_mlp_param_count(dim), np.float32)
        assert lib.vg_mlp_get_params(m, params.ctypes.data) == 0
        grads, loss, feats = _gradients(lib, m, q, valid, dim)
        ref_loss, ref = mlp.loss_and_gradients(params, feats, valid.cpu().numpy(), dim)
        assert abs(loss - ref_loss) <= 1e-5 * max(1.0, abs(ref_loss))
        got, want = mlp.split(grads, dim), mlp.split(ref, dim)
        for k in want:
            top = np.abs(want[k]).max()
            assert np.abs(got[k] - want[k]).max() <= 2e-3 * top + 1e-9, k
            assert np.linalg.norm(got[k] - want[k]) <= 1e-3 * np.linalg.norm(want[k]) + 1e-9, k
    finally:
        lib.vg_mlp_destroy(m)


@pytest.mark.parametrize("n,batch,dim", [(128, 128, 7), (1024, 512, 14), (1536, 768, 20)])
def test_adam_follows_the_gradients(n, batch, dim):
    """Steps of batch rows: each moves the weights as Adam does with the step's own gradients (taken
    from a second handle that holds the same weights), in float64 from float32 state: a few units
    of float32 rounding of the update's operations, 1e-6 of the weights plus 1e-4 of the step (1e-7)."""
    import torch

    from vamp_gb300._lib import lib

    q, valid = _inputs(n, dim, 5)
    count = lib.vg_mlp_param_count(dim)
    a, b = lib.vg_mlp_create(dim, 9), lib.vg_mlp_create(dim, 9)
    try:
        w = np.zeros(count, np.float32)
        lib.vg_mlp_get_params(a, w.ctypes.data)
        m, v = np.zeros(count), np.zeros(count)
        step = 0
        for off in range(0, n, batch):
            assert lib.vg_mlp_set_params(b, w.ctypes.data) == 0
            g, _, _ = _gradients(lib, b, q[off:off + batch], valid[off:off + batch], dim)
            assert lib.vg_mlp_train_device(a, q[off:off + batch].data_ptr(), valid[off:off + batch].data_ptr(), batch, 1, batch,
                                           1e-3, None, torch.cuda.current_stream().cuda_stream) == 0, lib.vg_last_error()
            step += 1
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g.astype(np.float64) ** 2
            want = w - 1e-3 * (m / (1 - 0.9 ** step)) / (np.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
            got = np.zeros(count, np.float32)
            lib.vg_mlp_get_params(a, got.ctypes.data)
            assert np.all(np.abs(got - want) <= 1e-6 * np.abs(want) + 1e-7)
            w = got
    finally:
        lib.vg_mlp_destroy(a)
        lib.vg_mlp_destroy(b)
