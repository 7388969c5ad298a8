"""Resources that make calls faster and are not to be had: calls then take
the way without them, with the same results.  (The refusals are made on the
host, _cuda_calls.py.)"""
import pytest

from _cuda_calls import run

pytestmark = pytest.mark.gpu

TEXTURE = """
arrays = scenes.displaced_spheres(60_000, 5, 64, 48, 3, env_w=64, env_h=32)
with _lib.Scene(arrays) as s:
    assert s.info().node_count >= 4096
    t = s.trace(scenes.random_rays(arrays, 20_000, seed=3))
    r = s.render(spp=2, max_depth=4, seed=1)
    with _lib.Batch([s, s]) as b:
        b.set_jobs([dict(scene=k, spp=2, max_depth=4, seed=k) for k in range(2)])
        b.render()
        o = [b.read(k) for k in range(2)]
    print(calls()[1], digest(*t[:3], r["beauty"], r["pathcount"], *(x["beauty"] for x in o)))
"""


def test_without_texture_objects(tmp_path):
    made, want = run(tmp_path, TEXTURE).split()
    assert int(made) == 2   # the scene's and the batch's
    none, got = run(tmp_path, TEXTURE, FAKE_NO_TEXTURE="1").split()
    assert int(none) == 0 and got == want
