"""er_batch_free waits for both of its streams before it releases what
launches on them read."""
import pytest

from _cuda_calls import run

pytestmark = pytest.mark.gpu

SCRIPT = """
arrays = scenes.displaced_spheres(60_000, 5, 64, 48, 3, env_w=64, env_h=32)
with _lib.Scene(arrays) as s:
    b = _lib.Batch([s])
    b.set_jobs([dict(scene=0, spp=8, max_depth=3, seed=k) for k in range(2)])
    t = A.er_batch_tuning()
    t.wave_paths = 64 * 48 * 2
    b.render(t)
    assert b.info()[0] >= 2
    at = len(calls()[2])
    b.close()
    print(calls()[2][at:])
"""


def test_streams_end_before_the_texture_goes(tmp_path):
    assert run(tmp_path, SCRIPT) == "SST"
