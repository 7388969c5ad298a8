"""er_scene_info.device_bytes counts the block that a scene keeps for host rays."""
import pytest

from eleven import _lib, scenes

pytestmark = pytest.mark.gpu


def test_kept_trace_block_is_counted():
    arrays = scenes.config0(x_res=8, y_res=8, n_spheres=4, subdiv=2)
    with _lib.Scene(arrays) as s:
        start = s.info().device_bytes
        s.trace(scenes.random_rays(arrays, 100, seed=1))
        for n in (30_000, 200_000):
            s.trace(scenes.random_rays(arrays, n, seed=n))
            assert 40 * n <= s.info().device_bytes - start <= 16 << 20
        kept = s.info().device_bytes
        s.trace(scenes.random_rays(arrays, 500_000, seed=2))   # 20 MB: a block of that call alone
        assert s.info().device_bytes == kept
