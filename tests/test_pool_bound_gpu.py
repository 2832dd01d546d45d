"""A context's pool holds what it keeps between calls and no more; buffers beyond that are allocated
one by one, and nothing of a result depends on where its buffers came from."""
import numpy as np
import pytest

import cases
from test_trace_gpu import make_scene

pytestmark = pytest.mark.gpu


def test_maps_beyond_the_pool(core, gpu_ctx):
    import torch

    keep = torch.cuda.mem_get_info()[1] // 64
    ctx = core.Context(0)
    rng = np.random.default_rng(3)
    pts = torch.from_numpy(rng.uniform(-1, 1, (200_000, 3)).astype(np.float32)).cuda()
    q = torch.from_numpy(rng.uniform(-1, 1, (1000, 3)).astype(np.float32)).cuda()

    def answers(m):
        idx, dist, count = m.build().knn(q, 10, 0.1)
        return idx.cpu(), dist.cpu(), count.cpu()

    def same(a, b):
        return all(torch.equal(x, y) for x, y in zip(a, b))

    first = core.PhotonMap.from_points(ctx, pts)  # from the pool
    want = answers(first)
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    n = int(keep * 0.9) // 64
    big = torch.rand(n, 3, device="cuda")
    maps = [core.PhotonMap.from_points(ctx, big) for _ in range(3)]  # 0.9 of the pool each
    small = [core.PhotonMap.from_points(ctx, pts) for _ in range(40)]  # 12.8 MB each: some on either side
    assert all(same(answers(m), want) for m in small)
    assert same(answers(maps[2]), answers(maps[0]))
    v, f = cases.soup(2000, 5)
    sc = make_scene(core, ctx, v, f)
    for m in maps + small:
        m.close()
    del big
    torch.cuda.empty_cache()
    # all but the pool's share is the device's again
    assert torch.cuda.mem_get_info()[0] >= before - keep - (256 << 20)
    assert same(answers(first), want)
    first.close()
    sc.close()
    ctx.close()
