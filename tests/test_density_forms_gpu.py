"""Photon density estimates by a warp, 16 lanes and 8 lanes per query (chosen by the number of queries): the
same points in calls of different sizes."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def maps(core, gpu_ctx):
    cfgs = importlib.import_module("2023_render_engine_b200.configs")
    scenes = importlib.import_module("2023_render_engine_b200.scenes")
    sc = core.Scene(gpu_ctx)
    (tv, tf), (sv, sf), _ = scenes.photon_terrain(seed=3, n=60)
    sc.set_materials(cfgs.cornell_materials())
    sc.add_mesh(tv, tf, material=0, shape_id=0)
    sc.add_mesh(sv, sf, material=0, shape_id=1)
    sc.add_point_light((-1.6, 2.6, 1.4), (1.0, 1.0, 1.0), 50.0)
    sc.commit()
    return {n: sc.trace_photons(n, max_depth=8, rr_depth=3, seed=5)[0].build() for n in (300, 20_000, 1_500_000)}, tv


@pytest.mark.parametrize("k", [1, 7, 64, 85, 86, 110, 111, 128])
@pytest.mark.parametrize("photons", [300, 20_000, 1_500_000])
def test_forms_agree(core, maps, photons, k):
    """Sums of at most k positive terms in another order: k roundings of 2^-24 each, twice."""
    pmap, tv = maps[0][photons], maps[1]
    N = importlib.import_module("2023_render_engine_b200._native")
    mat = core.material(N.RT_MAT_LAMBERTIAN, color=(0.6, 0.55, 0.45))
    rng = np.random.default_rng(k)
    n = 41_001
    pts = (tv[rng.integers(0, len(tv), n)] + rng.normal(0, 0.01, (n, 3))).astype(np.float32)
    wo = rng.normal(size=(n, 3)).astype(np.float32)
    wo[:, 1] = np.abs(wo[:, 1]) + 0.2
    wo /= np.linalg.norm(wo, axis=1, keepdims=True)
    nrm = np.tile(np.array([0, 1, 0], np.float32), (n, 1))
    sid = rng.integers(-1, 2, n).astype(np.int32)
    pts, nrm, wo, sid = (torch.from_numpy(a).cuda() for a in (pts, nrm, wo, sid))

    for radius in (100.0, 0.05, 1e-6):
        def density(q):
            return pmap.density(mat, pts[:q].contiguous(), nrm[:q].contiguous(), wo[:q].contiguous(), k, radius,
                                shape_dev=sid[:q].contiguous())

        want = density(499)
        for q in (1, 3, 6_000, 6_001, 10_001, 14_000, 14_001, 20_000, 40_000, 41_001):
            got = density(q)[:499]
            assert torch.isfinite(got).all()
            assert ((got - want[:q]).abs() <= 2 * (k + 2) * 2.0 ** -24 * want[:q].abs()).all()
    assert (density(499) == 0).float().mean() > 0.5  # hardly a photon that near
