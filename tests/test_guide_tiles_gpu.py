"""Gradient of the path guide at the edges of the training kernels' tiles: rows of one 128-row tile,
tiles of a block, 64-row stages and chunks of the weight gradient."""
import importlib

import numpy as np
import pytest

from oracle import guide_oracle as G

pytestmark = pytest.mark.gpu

LO, HI = np.array([-2.0, 0.0, -2.0], np.float32), np.array([2.0, 2.5, 2.0], np.float32)


@pytest.mark.parametrize("B", [1, 63, 64, 65, 127, 128, 129, 255, 257, 511, 1000, 37_889, 76_000])
def test_gradient_of_ragged_batches(core, gpu_ctx, B):
    """Against the oracle with FP16 operands. Its rounding order differs from the tensor core's: a
    half-precision step is 2^-11, some ten of them add up along the layers, and a sample whose ReLU
    changes sign adds its share; a row, column or lobe in the wrong place changes a layer's gradient
    by its own size. So each layer within 10%, and the same bits for the same batch."""
    import torch

    rng = np.random.default_rng(B)
    unit = lambda v: v / np.linalg.norm(v, axis=-1, keepdims=True)
    q = np.concatenate([rng.uniform(LO, HI, (B, 3)), unit(rng.normal(size=(B, 3))), unit(rng.normal(size=(B, 3)))],
                       1).astype(np.float32)
    wi = unit(rng.normal(size=(B, 3))).astype(np.float32)
    pdf, w = rng.uniform(0.05, 1, B).astype(np.float32), rng.lognormal(0, 1, B).astype(np.float32)
    g = core.Guide(gpu_ctx, LO, HI, learning_rate=1e-2, seed=7)
    p = g.params()
    p += rng.normal(0, 0.02, p.shape).astype(np.float32)  # biases too
    g.set_params(p)
    args = [torch.from_numpy(a.reshape(-1)).cuda() for a in (q, wi, pdf, w)]
    loss, grad = g.train_step(*args, apply=False, want_grad=True)
    ref_loss, ref = G.loss_and_grad(p, q, wi, pdf, w, LO, HI, fp16=True)
    assert abs(loss - ref_loss) <= 1e-2 * abs(ref_loss)
    for l, (wo, bo) in enumerate(G.OFFSETS):
        for a, b in ((wo, bo), (bo, bo + G.layer_out(l))):
            assert np.linalg.norm(grad[a:b] - ref[a:b]) <= 0.1 * np.linalg.norm(ref[a:b]), (l, a)
    assert np.array_equal(grad, g.train_step(*args, apply=False, want_grad=True)[1])
    g.close()


def test_raw_outputs_at_any_alignment(core, gpu_ctx):
    """Rows are written 16 bytes at a time where the buffer allows it: the same values one float on."""
    import ctypes
    import torch

    N = importlib.import_module("2023_render_engine_b200._native")
    rng = np.random.default_rng(2)
    B = 1001
    unit = lambda v: v / np.linalg.norm(v, axis=-1, keepdims=True)
    q = np.concatenate([rng.uniform(LO, HI, (B, 3)), unit(rng.normal(size=(B, 3))), unit(rng.normal(size=(B, 3)))],
                       1).astype(np.float32)
    g = core.Guide(gpu_ctx, LO, HI, learning_rate=1e-2, seed=7)
    qd = torch.from_numpy(q.reshape(-1)).cuda()
    want = g.eval(qd).reshape(-1)
    for shift in (1, 2, 3):
        out = torch.full((B * N.GUIDE_OUTPUTS + 8,), -7.0, device="cuda")
        N.check(N.lib().rt_guide_eval(g.handle, qd.data_ptr(), B, ctypes.c_void_p(out.data_ptr() + 4 * shift)))
        assert torch.equal(out[shift:shift + want.numel()], want)
        assert (out[:shift] == -7.0).all() and (out[shift + want.numel():] == -7.0).all()
    g.close()
