"""Nearest-neighbour queries on either side of the line between a thread and a group of lanes per query
(few neighbours of many queries): the same queries in one large call and in small ones."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes", [False, True])
@pytest.mark.parametrize("kind", ["scattered", "quantised"])
@pytest.mark.parametrize("k", [1, 2, 8, 9])
def test_thread_and_group_agree(core, gpu_ctx, k, kind, shapes):
    rng = np.random.default_rng(k)
    p = rng.uniform(-1, 1, (20_011, 3)).astype(np.float32)
    if kind == "quantised":  # equal distances, few equal coordinates at splits
        p[:, 1] = np.round(p[:, 1] * 4096) / 4096
    n = 25_000 * k  # the first count answered by threads, for k up to 8
    q = torch.from_numpy(rng.uniform(-1, 1, (n, 3)).astype(np.float32)).cuda()
    sid = torch.from_numpy(rng.integers(0, 3, len(p)).astype(np.int32)).cuda() if shapes else None
    qs = torch.from_numpy(rng.integers(-1, 3, n).astype(np.int32)).cuda() if shapes else None
    m = core.PhotonMap.from_points(gpu_ctx, torch.from_numpy(p).cuda(), sid).build()
    large = m.knn(q, k, 0.2, shape_dev=qs)
    step = 25_000 * k - 1 if k == 1 else 24_999
    for a in range(0, n, step):
        part = m.knn(q[a:a + step].contiguous(), k, 0.2, shape_dev=None if qs is None else qs[a:a + step].contiguous())
        for x, y in zip(part, large):
            assert torch.equal(x, y[a:a + step])
