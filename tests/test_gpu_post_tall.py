"""Bloom of very tall and very wide images (er_postprocess takes any sides up
to 2^28 pixels) against the oracle."""
import numpy as np
import pytest

import _oracle as O
from eleven import _abi as A
from eleven import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(3, 65_535 * 32), (3, 65_535 * 32 + 1), (33, 2_200_000), (2_200_000, 3)])
def test_bloom_of_long_images(w, h):
    rng = np.random.default_rng(w + h)
    img = np.zeros((w * h, 4), np.float32)
    lit = rng.integers(0, w * h, 100_000)
    img[lit] = rng.uniform(0.5, 4.0, (len(lit), 4)).astype(np.float32)
    o = A.er_post_opts(1.0, 0, 0, 0, 0, 0, 1.0, 0.4, 3.0)
    out, ldr = _lib.postprocess(img, w, h, bloom_threshold=1.0, bloom_power=0.4, bloom_radius=3.0)
    want = O.postprocess(img, w, h, o)
    assert np.array_equal(out.view(np.uint32), want.view(np.uint32))
    assert np.array_equal(ldr, _lib.encode_ldr(out, w, h))
