"""Camera rays: the offset of a sample within its pixel, evaluated in pairs of
floats, against the oracle's double expression, over resolutions and sensor
sizes (including sizes the pairs cannot hold, which take the double)."""
import numpy as np
import pytest

import _oracle as O
from eleven import _lib, scenes

pytestmark = pytest.mark.gpu


RES = [(1, 1), (7, 3), (320, 240), (641, 479), (1920, 1), (1, 1080)]


# (the oracle's unpruned traversal takes minutes for the rays of a huge sensor at a large resolution)
@pytest.mark.parametrize("res,sensor", [(r, s) for s in (0.035, 36.0, 1e-30, 0.0) for r in RES] +
                         [((1, 1), 3e37), ((7, 3), 3e37)])
@pytest.mark.parametrize("bokeh", [False, True])
def test_camera_rays_match_oracle(res, sensor, bokeh):
    """First-bounce outcomes depend on nothing but the camera rays: with depth
    1 every path's radiance and vertex count equals the oracle's, up to the
    last places of the environment lookup."""
    arrays = scenes.config0(x_res=res[0], y_res=res[1], n_spheres=3, subdiv=1)
    arrays.env = scenes.constant_env((0.5, 0.5, 0.5), size=16)
    arrays.camera.update(sensor_width=sensor, bokeh=bokeh, aperture=2.0, focus_distance=9.0)
    if sensor > 1:
        arrays.camera["focal_length"] = float(sensor)
    with _lib.Scene(arrays) as s:
        rad, b = s.render_paths(4, max_depth=1, seed=11)
    orc = O.OrcScene(arrays)
    orad, ob = orc.render_paths(4, max_depth=1, seed=11)
    orc.close()
    assert np.array_equal(b, ob.reshape(b.shape))
    orad = orad.reshape(rad.shape)
    fin = np.isfinite(orad)
    assert np.array_equal(np.isfinite(rad), fin)
    # same rays, same hits; the shading itself rounds as in the per-path parity tests
    assert np.isclose(rad[fin], orad[fin], rtol=1e-3, atol=1e-6).mean() > 0.999
