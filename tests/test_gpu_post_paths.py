"""The kernels of er_postprocess against the oracle where their tiles,
value ranges and buffer rules have edges."""
import ctypes as C

import numpy as np
import pytest
import torch

import _oracle as O
from eleven import _abi as A
from eleven import _lib

pytestmark = pytest.mark.gpu


def _opts(**kw):
    d = dict(exposure=1.0, tonemap=0, clamp=0, srgb=0, flip_x=0, flip_y=0, bloom_threshold=0.0, bloom_power=0.0,
             bloom_radius=0.0)
    d.update(kw)
    return d, A.er_post_opts(*d.values())


def _image(w, h, seed):
    rng = np.random.default_rng(seed)
    img = np.exp(rng.normal(-0.5, 1.5, (w * h, 4))).astype(np.float32)
    img[rng.random(w * h) < 0.3] = 0.0
    img[:, 3] = 1.0
    return img


def _same(a, b):
    return np.array_equal(a.view(np.uint32)[~np.isnan(b)], b.view(np.uint32)[~np.isnan(b)]) and np.array_equal(
        np.isnan(a), np.isnan(b))


# one tile, a pixel more and less, several; blur half-widths 1, 2, 4, the
# widest in shared memory (24) and the first beyond (25); images narrower than the blur
@pytest.mark.parametrize("w,h", [(1, 1), (31, 33), (32, 32), (33, 31), (65, 70), (130, 5), (5, 130)])
@pytest.mark.parametrize("radius", [2.0, 5.0, 9.0, 49.0, 50.0])
def test_bloom_tiles(w, h, radius):
    img = _image(w, h, w * 1000 + h)
    if w * h > 100:
        img[w * h // 2, 0] = np.inf   # an infinite pixel spreads as in the reference
    kw, o = _opts(exposure=1.3, bloom_threshold=1.0, bloom_power=0.4, bloom_radius=radius, flip_x=1)
    out, ldr = _lib.postprocess(img, w, h, **kw)
    want = O.postprocess(img, w, h, o)
    assert _same(out, want)
    assert np.array_equal(ldr, _lib.encode_ldr(out, w, h))


def test_bloom_threshold_and_dark_tiles():
    """Pixels whose mean is the threshold to the last bit, and tiles without a bright pixel."""
    w, h = 96, 64
    img = np.full((w * h, 4), 0.25, np.float32)
    img[: w * 20, :3] = np.float32(1.0)
    step = np.arange(w * 20, dtype=np.uint32) % 5
    img[: w * 20, 1] = (np.float32(1.0).view(np.uint32) + step - 2).view(np.float32)
    kw, o = _opts(bloom_threshold=1.0, bloom_power=0.4, bloom_radius=5.0)
    out, _ = _lib.postprocess(img, w, h, **kw)
    assert _same(out, O.postprocess(img, w, h, o))


@pytest.mark.parametrize("tonemap,srgb", [(A.ER_TONEMAP_ACES, 0), (A.ER_TONEMAP_ACES, 1), (A.ER_TONEMAP_NONE, 1)])
def test_channels_over_the_float_range(tonemap, srgb):
    """Values of every magnitude, negative, denormal, infinite and NaN."""
    rng = np.random.default_rng(7)
    bits = rng.integers(0, 1 << 32, 4 * 256 * 64, dtype=np.uint64).astype(np.uint32)
    img = bits.view(np.float32).copy()
    n = len(img) // 2
    img[:n] = np.float32(2.0) ** rng.uniform(-24, 12, n).astype(np.float32)   # the range of a film
    img[:8] = [0.0, -0.0, 1.0, np.inf, -np.inf, np.nan, 1e-45, 0.5]
    img = img.reshape(-1, 4)
    kw, o = _opts(tonemap=tonemap, srgb=srgb)
    out, ldr = _lib.postprocess(img, 256, 64, **kw)
    want = O.postprocess(img, 256, 64, o)
    fin = np.isfinite(want)
    # (the power in double rounds 1 ulp apart on the host's libm)
    np.testing.assert_array_max_ulp(out[fin], want[fin], maxulp=1 if srgb else 0)
    assert np.array_equal(np.isnan(out), np.isnan(want))
    assert np.array_equal(ldr, _lib.encode_ldr(out, 256, 64))


@pytest.mark.parametrize("kw", [dict(exposure=1.5, clamp=1), dict(flip_x=1), dict(flip_y=1, srgb=1, clamp=1),
                                dict(bloom_threshold=1.0, bloom_power=0.3, bloom_radius=9.0)])
@pytest.mark.parametrize("where", ["in place", "shifted", "bytes over the input"])
def test_outputs_over_the_input(kw, where):
    """Device outputs that overlap the input give the result of separate buffers."""
    w, h = 70, 45
    n = w * h
    img = _image(w, h, 3)
    kw, o = _opts(**kw)
    out, ldr = _lib.postprocess(img, w, h, **kw)
    buf = torch.zeros(2 * n * 4, dtype=torch.float32, device="cuda")
    bytes_ = torch.zeros(n * 4, dtype=torch.uint8, device="cuda")
    buf[: n * 4] = torch.from_numpy(img.reshape(-1)).cuda()
    base = buf.data_ptr()
    dst = {"in place": base, "shifted": base + 16 * 100, "bytes over the input": base + 16 * n}[where]
    d_ldr = base + 64 if where == "bytes over the input" else bytes_.data_ptr()
    torch.cuda.synchronize()
    _lib.check(_lib.load().er_postprocess(C.c_void_p(base), w, h, C.byref(o), C.c_void_p(dst), C.c_void_p(d_ldr),
                                          A.ER_RENDER_DEVICE_OUT), "er_postprocess")
    got = buf.cpu().numpy()[(dst - base) // 4:][: n * 4].reshape(n, 4)
    assert _same(got, out)
    got_ldr = buf.cpu().numpy().view(np.uint8)[64: 64 + 4 * n] if where == "bytes over the input" else bytes_.cpu().numpy()
    assert np.array_equal(got_ldr.reshape(-1), ldr.reshape(-1))
