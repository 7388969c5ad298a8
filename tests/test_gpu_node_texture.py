"""Reading half of the FP32 node planes through the texture unit (trees of 4096
nodes on) changes no hit: against the counting kernels, which read every plane
with plain loads, below and above that size, for both builders, in a batch
whose merged nodes lie behind another scene's, and in films."""
import numpy as np
import pytest

from eleven import _abi as A
from eleven import _lib, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_tris", [20_000, 40_000, 120_000])
@pytest.mark.parametrize("builder", [A.ER_BUILDER_HOST, A.ER_BUILDER_GPU])
def test_hits(n_tris, builder):
    arrays = scenes.displaced_spheres(n_tris, 3, 64, 48, 2, env_w=32, env_h=16)
    with _lib.Scene(arrays, builder=builder) as s:
        nodes = s.info().node_count
        assert (nodes >= 4096) == (n_tris > 30_000)
        rays = scenes.random_rays(arrays, 100_003, seed=1)
        got, plain = s.trace(rays), s.trace(rays, stats=True)
        for a, b in zip(got[:3], plain[:3]):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
        assert (got[0] >= 0).sum() > 1000
        # camera, bounce and both kinds of shadow rays
        film = s.render(2, max_depth=4, seed=5)
        counted = s.render(2, max_depth=4, seed=5, flags=A.ER_RENDER_COUNT)
        for k in ("beauty", "samples", "pathcount"):
            assert np.array_equal(film[k], counted[k], equal_nan=True)


def test_batch_and_lifetime():
    """The batch's nodes have a texture of their own; scenes freed and made
    again in any order do not disturb one another's."""
    big = scenes.displaced_spheres(60_000, 3, 64, 48, 2, env_w=32, env_h=16)
    small = scenes.displaced_spheres(5_000, 4, 40, 30, 1, env_w=32, env_h=16)
    for order in ([big, small], [small, big], [big, big]):
        ss = [_lib.Scene(a) for a in order]
        want = [s.render(2, max_depth=4, seed=7 + k)["beauty"] for k, s in enumerate(ss)]
        with _lib.Batch(ss) as b:
            b.set_jobs([dict(scene=k, spp=2, max_depth=4, seed=7 + k) for k in range(2)])
            for _ in range(2):
                b.render()
            for k in range(2):
                assert np.array_equal(b.read(k)["beauty"], want[k], equal_nan=True)
        ss[0].close()
        assert np.array_equal(ss[1].render(2, max_depth=4, seed=8)["beauty"], want[1], equal_nan=True)
        ss[1].close()
