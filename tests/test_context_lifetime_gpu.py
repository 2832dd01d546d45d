"""A context's objects outlive its handle, in whatever order they are let go of (a garbage collector
finalises the context before its scenes), and contexts side by side keep their memory apart."""
import gc
import itertools

import numpy as np
import pytest

import cases
from test_trace_gpu import S, make_scene, trace_gpu

pytestmark = pytest.mark.gpu


def objects(core, ctx):
    import torch

    v, f = cases.soup(500, 2)
    sc = make_scene(core, ctx, v, f)
    pts = torch.from_numpy(np.random.default_rng(1).uniform(-1, 1, (5000, 3)).astype(np.float32)).cuda()
    return [sc, core.PhotonMap.from_points(ctx, pts).build(), core.Guide(ctx, [-1] * 3, [1] * 3, seed=1)]


def use(core, objs):
    import torch

    o, d = S.random_rays(2000, seed=4, lo=-1.0, hi=1.0)
    ids, t, _ = trace_gpu(objs[0], o, d)
    q = torch.from_numpy(np.ascontiguousarray(o[:64])).cuda()
    idx, dist, count = objs[1].knn(q, 8, 10.0)
    rows = torch.cat([q, torch.nn.functional.normalize(q + 2.0), torch.nn.functional.normalize(q - 2.0)], 1).contiguous()
    return [ids, t, idx.cpu().numpy(), dist.cpu().numpy(), objs[2].eval(rows).cpu().numpy()]


@pytest.mark.parametrize("order", list(itertools.permutations(range(3))))
def test_objects_outlive_their_context(core, gpu_ctx, order):
    want = use(core, objects(core, gpu_ctx))
    ctx = core.Context(0)
    objs = objects(core, ctx)
    ctx.close()
    for k in range(3):
        got = use(core, objs) if k == 0 else None
        if got is not None:
            assert all(np.array_equal(a, b) for a, b in zip(got, want))
        objs[order[k]].close()


def test_collected_after_their_context(core, gpu_ctx):
    class Holder:
        pass

    h = Holder()
    h.ctx = core.Context(0)  # the oldest of the cycle: its finaliser runs first
    h.objs = objects(core, h.ctx)
    h.self = h
    del h
    gc.collect()
    assert np.isfinite(use(core, objects(core, gpu_ctx))[4]).all()


def test_contexts_side_by_side(core, gpu_ctx):
    a, b = core.Context(0), core.Context(0)
    oa, ob = objects(core, a), objects(core, b)
    want = use(core, oa)
    assert all(np.array_equal(x, y) for x, y in zip(use(core, ob), want))
    for x in oa:
        x.close()
    a.close()  # its pool is given back; the other context's objects stay
    oc = objects(core, b)
    for o in (ob, oc):
        assert all(np.array_equal(x, y) for x, y in zip(use(core, o), want))


def test_pool_is_given_back_to_an_allocation_that_fails(core, gpu_ctx):
    """What one context's pool keeps between calls serves another whose allocation finds no memory."""
    import torch

    a, b = core.Context(0), core.Context(0)
    pts = torch.rand(4_000_000, 3, device="cuda")
    core.PhotonMap.from_points(a, pts).build().close()  # 256 MB of photons and 400 MB of workspace stay in a's pool
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - (200 << 20), dtype=torch.uint8, device="cuda")
    try:
        m = core.PhotonMap.from_points(b, pts)  # 256 MB, of which 200 are free
        m.build()
        idx, _, count = m.knn(pts[:100].contiguous(), 1, 10.0)
        assert (count == 1).all() and torch.equal(idx[:, 0].cpu(), torch.arange(100, dtype=torch.int32))
        m.close()
    finally:
        del hog
        torch.cuda.empty_cache()
