"""er_trace_closest on host arrays: the blocks a scene keeps between calls give
the results of device pointers at every size class, growing and shrinking,
with and without the optional outputs, from several scenes and threads."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from eleven import _abi as A
from eleven import _lib, scenes

pytestmark = pytest.mark.gpu

# 40 bytes a ray: page-locked up to 2^19 bytes, in a kept device block up to 2^24, then in one of the call alone
SIZES = [1, 63, 65, 13_056, 13_200, 5, 26_300, 419_000, 420_000, 100, 30_000]


def _p(a):
    return None if a is None else C.c_void_p(a.data_ptr() if isinstance(a, torch.Tensor) else a.ctypes.data)


def _call(scene, rays, dist, uv, device):
    n = len(rays)
    if device:
        r = torch.from_numpy(rays).cuda()
        out = [torch.full((n,), -7, dtype=torch.int32, device="cuda"),
               torch.zeros(n, device="cuda") if dist else None, torch.zeros((n, 2), device="cuda") if uv else None]
        torch.cuda.synchronize()
    else:
        r = rays
        out = [np.full(n, -7, np.int32), np.zeros(n, np.float32) if dist else None,
               np.zeros((n, 2), np.float32) if uv else None]
    _lib.check(_lib.load().er_trace_closest(scene.h, _p(r), n, *(_p(o) for o in out),
                                            A.ER_TRACE_DEVICE_PTRS if device else 0, None), "er_trace_closest")
    return [o.cpu().numpy() if isinstance(o, torch.Tensor) else o for o in out]


def _equal(a, b):
    return all((x is None and y is None) or np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(a, b))


@pytest.mark.parametrize("dist,uv", [(True, True), (True, False), (False, True), (False, False)])
def test_host_arrays_match_device_arrays(dist, uv):
    arrays = scenes.config0(x_res=8, y_res=8, n_spheres=4, subdiv=2)
    with _lib.Scene(arrays) as s:
        for n in SIZES:
            rays = scenes.random_rays(arrays, n, seed=n)
            assert _equal(_call(s, rays, dist, uv, False), _call(s, rays, dist, uv, True)), n


def test_scenes_in_threads():
    """Each handle has its own blocks."""
    arrays = [scenes.config0(x_res=8, y_res=8, seed=k, n_spheres=4, subdiv=2) for k in range(3)]
    ss = [_lib.Scene(a) for a in arrays]
    rays = [scenes.random_rays(a, 20_000, seed=9) for a in arrays]
    want = [_call(s, r, True, True, True) for s, r in zip(ss, rays)]
    bad = []

    def work(k):
        for _ in range(20):
            if not _equal(_call(ss[k], rays[k], True, True, False), want[k]):
                bad.append(k)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    [s.close() for s in ss]
    assert not bad
