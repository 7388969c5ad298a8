"""How work is split over the GPU changes no result: rays per warp of small
trace queues, and the order of paths within a wave, at the sizes where the
splits have remainders."""
import numpy as np
import pytest

import _oracle as O
from eleven import _abi as A
from eleven import _lib, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def small():
    arrays = scenes.config0(x_res=64, y_res=48, n_spheres=6, subdiv=2)
    return arrays, _lib.Scene(arrays), O.OrcScene(arrays)


# one ray, the fewest rays of a warp (4) and its neighbours, one warp, one
# block, and both sides of 4 rays per resident warp (152 SMs x 28 warps x 4)
@pytest.mark.parametrize("n", [1, 3, 4, 5, 31, 33, 129, 17023, 17025, 68096, 272385])
def test_small_trace_queues(small, n):
    arrays, scene, orc = small
    rays = scenes.random_rays(arrays, n, seed=n)
    tri, dist, _, _ = scene.trace(rays)
    rtri, rdist = orc.trace(rays)
    bad = np.nonzero(tri != rtri)[0]
    assert all(dist[i] == rdist[i] for i in bad)  # exact distance ties only
    ok = tri == rtri
    assert np.array_equal(dist[ok].view(np.uint32), rdist[ok].view(np.uint32))


# whole tiles; remainders in x, in y, in both; smaller than a tile; a last
# group of one, two and three pixels
@pytest.mark.parametrize("w,h", [(16, 8), (13, 8), (16, 7), (13, 7), (7, 3), (1, 1), (9, 1), (3, 2), (37, 19)])
@pytest.mark.parametrize("spp", [1, 3])
def test_path_order(w, h, spp):
    arrays = scenes.config0(x_res=w, y_res=h, n_spheres=4, subdiv=1)
    with _lib.Scene(arrays) as s:
        # every path against the oracle's (the numbers depend on pixel and sample alone)
        rad, bounces = s.render_paths(spp, max_depth=3, seed=5)
        orc = O.OrcScene(arrays)
        orad, ob = orc.render_paths(spp, max_depth=3, seed=5)
        orc.close()
        assert np.array_equal(bounces, ob.reshape(bounces.shape))
        close = np.isclose(rad, orad.reshape(rad.shape), rtol=1e-3, atol=1e-6)
        assert close.mean() > 0.99
        # the film is the same however the samples are cut into waves
        whole = s.render(spp, max_depth=3, seed=5, spp_per_wave=spp, flags=A.ER_RENDER_ONE_STREAM, aov=True)
        for k in range(1, spp + 1):
            cut = s.render(spp, max_depth=3, seed=5, spp_per_wave=k, aov=True)
            for key in ("beauty", "normal", "samples", "pathcount"):
                assert np.array_equal(cut[key], whole[key], equal_nan=True), (k, key)
        assert (whole["samples"] <= spp).all()


def test_shade_groups():
    """Waves of 0.3, 1.5 and 4.9 million paths (shade groups of 128 to 512 items) give the same film."""
    arrays = scenes.config0(x_res=640, y_res=480)
    with _lib.Scene(arrays) as s:
        whole = s.render(16, max_depth=4, seed=2, spp_per_wave=16)
        for k in (1, 5):
            cut = s.render(16, max_depth=4, seed=2, spp_per_wave=k)
            for key in ("beauty", "samples", "pathcount"):
                assert np.array_equal(cut[key], whole[key], equal_nan=True), (k, key)


def test_gradient_shade_groups():
    """Gradient waves of 2.5 million paths (shade groups of 8 x 128 items) against the sum over calls whose waves
    have 0.6 and 0.3 million (2 x 128, 128).  A sum of n floats in another order differs by about sqrt(n) 2^-24 of
    the sum of their absolute values: 6e-5 for the million terms of a material, less for a texel; an item left out
    or taken twice changes its texels by a hundredth."""
    arrays = scenes.config0(x_res=640, y_res=480)
    with _lib.Scene(arrays) as s:
        out = s.render(16, max_depth=3, seed=4)
        d = np.zeros_like(out["beauty"])
        d[:, :3] = 1.0
        whole = s.backward(16, d, out["samples"], max_depth=3, seed=4)[:2]
        assert all(np.abs(g).max() > 0 for g in whole)
        for k in (1, 4):
            parts = [s.backward(k, d, out["samples"], max_depth=3, seed=4, sample_begin=b)[:2] for b in range(0, 16, k)]
            for i in (0, 1):
                g = np.stack([p[i] for p in parts]).astype(np.float64)
                bound = 1e-4 * np.abs(g).sum(0) + 1e-6 * np.abs(whole[i]).max()
                assert (np.abs(g.sum(0) - whole[i]) <= bound).all(), (k, i)
