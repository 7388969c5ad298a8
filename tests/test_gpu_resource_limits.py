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

TRACE = """
arrays = scenes.config0(x_res=8, y_res=8, n_spheres=4, subdiv=2)
with _lib.Scene(arrays) as s:
    r = s.render(spp=1, max_depth=3, seed=1)
    t = [s.trace(scenes.random_rays(arrays, n, seed=n))[:3] for n in (1, 63, 5_000, 13_056, 20_000)]
    print(calls()[0], digest(r["beauty"], *(x for k in t for x in k)))
"""


def test_without_page_locked_memory_for_rays(tmp_path):
    held, want = run(tmp_path, TRACE).split()
    assert int(held) >= 1 << 19
    few, got = run(tmp_path, TRACE, FAKE_HOST_MAX="4096").split()
    assert int(few) <= 4096 and got == want


MANY = """
arrays = scenes.config0(x_res=8, y_res=8, n_spheres=1, subdiv=0)
rays = scenes.random_rays(arrays, 100, seed=1)
ss = [_lib.Scene(arrays) for k in range(80)]
most = calls()[0]
d = {digest(*s.trace(rays)[:3]) for s in ss}
[s.close() for s in ss]
none = calls()[0]
ss = [_lib.Scene(arrays)]
again = calls()[0]
d.add(digest(*ss[0].trace(rays)[:3]))
ss[0].close()
print(most, none, again, calls()[0], len(d))
"""


def test_page_locked_memory_of_many_scenes(tmp_path):
    """Bounded over all scenes, given back, and had again by a later scene."""
    most, none, again, end, results = map(int, run(tmp_path, MANY).split())
    assert most <= (1 << 24) + 80 * 4096
    assert none == 0 and end == 0 and again >= 1 << 19
    assert results == 1
