"""Nearest-neighbour queries of traced photon maps, whose tree is built on the GPU and differs from the
host's where a split coordinate occurs twice: the answers are those of the host's tree, which is built
only once a query meets equal distances."""
import importlib
import time

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def traced(core, gpu_ctx):
    """A traced map of the photon scene, not built, and its photons as a point set."""
    cfgs = importlib.import_module("2023_render_engine_b200.configs")
    scenes = importlib.import_module("2023_render_engine_b200.scenes")
    sc = core.Scene(gpu_ctx)
    (tv, tf), _, _ = scenes.photon_terrain(seed=3, n=100)
    sc.set_materials(cfgs.cornell_materials())
    sc.add_mesh(tv, tf, material=0, shape_id=0)
    sc.add_point_light((-1.6, 2.6, 1.4), (1.0, 1.0, 1.0), 50.0)
    sc.commit()

    def trace():
        return sc.trace_photons(1_000_000, max_depth=8, rr_depth=3, seed=5)[0]

    pos = np.ascontiguousarray(trace().photons()["pos"], dtype=np.float32)
    return trace, torch.from_numpy(pos).cuda()


@pytest.mark.parametrize("k", [1, 5, 50, 128])
def test_answers_are_those_of_the_host_tree(core, gpu_ctx, traced, k):
    trace, pts = traced
    assert pts.shape[0] > 100_000
    host = core.PhotonMap.from_points(gpu_ctx, pts).build()
    m = trace().build()
    rng = np.random.default_rng(k)
    p = pts.cpu().numpy()
    pairs = p[rng.integers(0, len(p), (20_000, 2))]
    # random points, points halfway between two photons (equal distances, up to rounding), photons
    q = np.concatenate([rng.uniform(-4, 4, (80_000, 3)).astype(np.float32), (pairs[:, 0] + pairs[:, 1]) * np.float32(0.5),
                        pairs[:1000, 0]]).astype(np.float32)
    q = torch.from_numpy(np.ascontiguousarray(q)).cuda()
    want = host.knn(q, k, 100.0)
    for _ in range(2):  # the call that finds the first equal distances, and one that has the host's tree
        for a, b in zip(m.knn(q, k, 100.0), want):
            assert torch.equal(a, b)
    m.build()  # a second build starts over
    for a, b in zip(m.knn(q, k, 100.0), want):
        assert torch.equal(a, b)


def test_no_host_tree_without_equal_distances(core, gpu_ctx, traced):
    trace, pts = traced
    m = trace().build()
    t0 = time.perf_counter()
    host = core.PhotonMap.from_points(gpu_ctx, pts).build()  # equal coordinates: includes a host build
    host_build = time.perf_counter() - t0
    q = torch.tensor([[0.1234, 0.5, 0.4321]], device="cuda")
    first = host.knn(q, 1, 100.0)
    t0 = time.perf_counter()
    got = m.knn(q, 1, 100.0)
    assert time.perf_counter() - t0 < 0.25 * host_build
    assert torch.equal(got[0], first[0]) and torch.equal(got[1], first[1])
