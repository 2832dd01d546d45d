"""The photon map's kd-tree build and its queries at the edges of the device build's ranges."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# a block finishes ranges of 1024 positions
SIZES = [1, 2, 3, 4, 63, 64, 65, 1023, 1024, 1025, 2047, 2048, 2049, 2051, 5000, 70_001]


def _points(n, kind, rng):
    """distinct: no coordinate occurs twice; lattice: many do, and whole points too; wide: one axis
    of no extent, one that reaches the largest floats."""
    if kind == "distinct":
        return np.stack([(rng.permutation(n) - n // 2) / 1024 for _ in range(3)], 1).astype(np.float32)
    if kind == "lattice":
        return rng.integers(-3, 4, (n, 3)).astype(np.float32) / 4
    p = rng.uniform(-1, 1, (n, 3)).astype(np.float32)
    p[:, 1] = 0.25
    p[: n // 3, 0] *= np.float32(3e38)
    return p


def _distances(p, q):
    with np.errstate(over="ignore"):
        d = q[:, None, :] - p[None, :, :]
        s = d * d
        return np.sqrt((s[..., 0] + s[..., 1]) + s[..., 2])


@pytest.mark.parametrize("kind", ["distinct", "lattice", "wide"])
@pytest.mark.parametrize("n", SIZES)
def test_nearest_neighbours_are_exact(core, gpu_ctx, n, kind):
    """Distances and counts are those of a search over all points, in the same 32-bit operations;
    each returned photon lies at its distance, and none is returned twice."""
    rng = np.random.default_rng(n)
    p = _points(n, kind, rng)
    q = p[rng.integers(0, n, 40)] + rng.normal(0, 0.02, (40, 3)).astype(np.float32)
    q[:4] = p[:4] if n >= 4 else p[0]
    d = _distances(p, q)
    m = core.PhotonMap.from_points(gpu_ctx, torch.from_numpy(p).cuda()).build()
    for k, radius in [(1, 100.0), (7, 0.5), (50, 1000.0), (128, np.inf)]:
        idx, dist, cnt = (t.cpu().numpy() for t in m.knn(torch.from_numpy(q).cuda(), k, radius))
        for i in range(len(q)):
            want = np.sort(d[i][d[i] < np.float32(radius)])[:k]
            assert cnt[i] == len(want)
            assert np.array_equal(dist[i, :cnt[i]], want)
            assert np.isinf(dist[i, cnt[i]:]).all() and (idx[i, cnt[i]:] == -1).all()
            assert np.array_equal(d[i][idx[i, :cnt[i]]], want)
            assert len(set(idx[i, :cnt[i]].tolist())) == cnt[i]
    m.close()


def test_points_that_are_not_finite_are_never_found(core, gpu_ctx):
    rng = np.random.default_rng(5)
    p = rng.uniform(-1, 1, (3000, 3)).astype(np.float32)
    p[::7, 1] = np.inf
    q = rng.uniform(-1, 1, (50, 3)).astype(np.float32)
    m = core.PhotonMap.from_points(gpu_ctx, torch.from_numpy(p).cuda()).build()
    idx, _, cnt = (t.cpu().numpy() for t in m.knn(torch.from_numpy(q).cuda(), 20, 100.0))
    assert (cnt == 20).all() and (idx % 7 != 0).all()
