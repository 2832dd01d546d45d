"""The bias gradient's sums over a batch, against the 64-bit sum of the gradients of its pieces of 8 rows (all
weights 1, so that a row's share does not depend on the batch)."""
import numpy as np
import pytest

from oracle import guide_oracle as G

pytestmark = pytest.mark.gpu

LO, HI = np.array([-2.0, 0.0, -2.0], np.float32), np.array([2.0, 2.5, 2.0], np.float32)


@pytest.mark.parametrize("B", [8, 64, 72, 256, 264, 1000, 4096])
def test_bias_gradient_is_the_sum_of_its_rows(core, gpu_ctx, B):
    """Every rounding of a 32-bit addition is at most 2^-24 of the sum of magnitudes: 3 levels over the 8 rows
    of a piece and 3 over the 8 pieces of a stage, the stages of a chunk, the chunks, and 4 for the scale
    (twice: the pieces' gradients have the same, with one stage and one chunk)."""
    import torch

    rng = np.random.default_rng(B)
    unit = lambda v: v / np.linalg.norm(v, axis=-1, keepdims=True)
    q = np.concatenate([rng.uniform(LO, HI, (B, 3)), unit(rng.normal(size=(B, 3))), unit(rng.normal(size=(B, 3)))],
                       1).astype(np.float32)
    wi = unit(rng.normal(size=(B, 3))).astype(np.float32)
    pdf = rng.uniform(0.05, 1, B).astype(np.float32)
    net = core.Guide(gpu_ctx, LO, HI, learning_rate=1e-2, seed=11)
    p = net.params()
    p += rng.normal(0, 0.02, p.shape).astype(np.float32)
    net.set_params(p)
    q, wi, pdf, w = (torch.from_numpy(a).cuda() for a in (q, wi, pdf, np.ones(B, np.float32)))

    def grad(a, b):
        part = [x[a:b].contiguous().reshape(-1) for x in (q, wi, pdf, w)]
        return np.asarray(net.train_step(*part, apply=False, want_grad=True)[1], np.float64)

    biases = np.concatenate([np.arange(bo, bo + G.layer_out(l)) for l, (_, bo) in enumerate(G.OFFSETS)])
    pieces = np.stack([grad(a, a + 8)[biases] * 8 for a in range(0, B, 8)])
    full = grad(0, B)[biases] * B
    padded = -(-B // 128) * 128
    chunk = max(256, -(-padded // 148 // 64) * 64)
    adds = 3 + 3 + chunk // 64 + -(-padded // chunk) + 4 + (3 + 3 + 1 + 1 + 4)
    assert np.abs(pieces).max() > 0
    assert (np.abs(full - pieces.sum(0)) <= adds * 2.0 ** -24 * np.abs(pieces).sum(0)).all()
    net.close()
