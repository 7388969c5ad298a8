"""The device builder's treelet and collapse kernels at the sizes where they
change course: fewer triangles than a treelet has leaves, a warp, a block and
their neighbours, equal centroids, and chains many levels deep."""
import dataclasses

import numpy as np
import pytest

from eleven import _abi as A
from eleven import _lib, scenes

pytestmark = pytest.mark.gpu


def _subset(arrays, n):
    return dataclasses.replace(arrays, positions=arrays.positions[:n], normals=arrays.normals[:n],
                               uvs=arrays.uvs[:n], tri_object=arrays.tri_object[:n])


def _nested(n, ratio):
    """n triangles with one centroid, each `ratio` times the size of the one
    before: the cheapest tree is a chain."""
    base = scenes.config0(x_res=8, y_res=8, n_spheres=1, subdiv=0)
    t = np.array([[1, 0, 0], [-0.5, 0.8, 0.1], [-0.5, -0.8, -0.1]], np.float32)
    s = (ratio ** np.arange(n)).astype(np.float32)
    pos = (t[None] * s[:, None, None]).astype(np.float32)
    return dataclasses.replace(base, positions=pos, normals=np.zeros_like(pos), uvs=np.zeros((n, 3, 2), np.float32),
                               tri_object=np.zeros(n, np.int32))


def _check(arrays, leaf=0):
    rays = scenes.random_rays(arrays, 20_000, seed=4)
    with _lib.Scene(arrays, max_leaf=leaf) as host, _lib.Scene(arrays, builder=A.ER_BUILDER_GPU, max_leaf=leaf) as dev:
        want, got = host.trace(rays), dev.trace(rays)
        info = dev.info()
    for a, b in zip(got[:3], want[:3]):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    assert (want[0] >= 0).any()
    return info


@pytest.mark.parametrize("n", [1, 2, 3, 4, 6, 7, 8, 9, 31, 32, 33, 127, 129, 2000])
@pytest.mark.parametrize("leaf", [1, 4])
def test_sizes(n, leaf):
    info = _check(_subset(scenes.config0(x_res=8, y_res=8, n_spheres=8, subdiv=2), n), leaf)
    assert info.tri_count == n
    assert info.leaf_count >= -(-n // max(leaf, 1))


@pytest.mark.parametrize("n,ratio", [(7, 2.0), (40, 1.5), (90, 1.2)])
def test_nested_chains(n, ratio):
    _check(_nested(n, ratio), 1)


def test_more_levels_than_one_batch_of_launches():
    """A chain of more than 16 levels of 4-wide nodes."""
    info = _check(_nested(70, 1.3), 1)
    assert 16 < info.bvh_depth <= 31
