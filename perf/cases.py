"""Workloads of the path tracer, each through the entry points a program calls.

listed() names the fixed ones, draw() makes more of the same ranges, prepare() builds what a program holds before the
call (scene handles, parameters, output buffers), run() is one pass, work() the bytes and operations it cannot do
without, exact() its result in 64-bit arithmetic where that can be had directly.

Scenes are the generators of eleven.scenes: icospheres on a ground quad ("small"), displaced and textured spheres
under a 2048x1024 environment with a sun ("film"), untextured displaced spheres under a 512x256 environment
("spheres"), icospheres under a 256x128 environment ("diff").  Their geometry depends on the case alone and is made
once per process; materials, lights, environment, camera and random numbers come from the seed.
"""
import ctypes as C
import dataclasses
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tfg-pathtracer_gb300"))

from eleven import _abi as A  # noqa: E402
from eleven import _lib, adjoint, scenes  # noqa: E402


def listed():
    return [
        # an interactive preview: one sample per pixel of a small scene into the caller's device film
        dict(name="preview_320x240", kind="render", scene="small", tris=20_000, width=320, height=240, spp=1, depth=5,
             bvh="fp32", aov=False, alias=False, fp64=False, out="device"),
        # a final frame: 1080p, thin lens, textures, sun, full depth (the benchmark's scene)
        dict(name="film_1080p_16spp", kind="render", scene="film", tris=1_180_000, width=1920, height=1080, spp=16,
             depth=8, bvh="fp32", aov=False, alias=False, fp64=False, out="device"),
        # progressive display: one sample per pixel and the film read back to page-locked host memory each call
        dict(name="progressive_1080p", kind="render", scene="film", tris=1_180_000, width=1920, height=1080, spp=1,
             depth=8, bvh="fp32", aov=False, alias=False, fp64=False, out="host"),
        # the options together, at a ragged size: 8-bit nodes, AOV passes, alias-table sampling, FP64 sums
        dict(name="q8_aov_641x479", kind="render", scene="spheres", tris=60_000, width=641, height=479, spp=9, depth=5,
             bvh="q8", aov=True, alias=True, fp64=True, out="device"),
        # a thumbnail from a caller that may not allocate while it renders
        dict(name="noalloc_200x150", kind="noalloc", scene="small", tris=20_000, width=200, height=150, spp=4, depth=5),
        # closest-hit queries in bulk on device arrays (visibility, picking grids, collision sweeps)
        dict(name="trace_1m", kind="trace", scene="spheres", tris=400_000, rays=1_000_003, bvh="fp32", out="device"),
        # a few queries from host arrays
        dict(name="trace_4099_host", kind="trace", scene="small", tris=20_000, rays=4_099, bvh="fp32", out="host"),
        # one optimisation step of the differentiation workload: parameters set, forward, loss, backward
        dict(name="adjoint_512", kind="adjoint", objects=64, width=512, height=512, spp=64, depth=6),
        # the same at the size of a quick fit
        dict(name="adjoint_129x97", kind="adjoint", objects=16, width=129, height=97, spp=16, depth=4),
        # many views of many scenes rendered together
        dict(name="batch_12", kind="batch", jobs=12, tris=60_000, spp=16, bvh="q8"),
        # tone map, bloom and 8-bit encoding of a finished frame
        dict(name="post_1080p_bloom", kind="post", width=1920, height=1080, bloom_radius=9.0, tonemap=2, srgb=True),
        # a changed scene: built with the device builder, then queried
        dict(name="build_300k", kind="build", tris=300_000, rays=20_000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "render", "noalloc", "trace", "adjoint", "batch", "post", "build"])
    if kind == "render":
        scene = rng.choice(["small", "spheres", "film"])
        w = _log(rng, 160, 1920)
        h = max(90, min(1080, int(w * rng.uniform(0.5, 0.8))))
        return dict(kind=kind, scene=scene, tris={"small": 20_000, "film": _log(rng, 100_000, 1_180_000),
                                                  "spheres": _log(rng, 10_000, 500_000)}[scene],
                    width=w, height=h, spp=max(1, min(_log(rng, 1, 32), 33_000_000 // (w * h))),
                    depth=rng.randint(3, 8), bvh=rng.choice(["fp32", "q8"]), aov=rng.random() < 0.3,
                    alias=rng.random() < 0.3, fp64=rng.random() < 0.3, out=rng.choice(["device", "host"]))
    if kind == "noalloc":
        return dict(kind=kind, scene=rng.choice(["small", "spheres"]), tris=20_000, width=rng.randint(64, 256),
                    height=rng.randint(48, 256), spp=_log(rng, 1, 16), depth=rng.randint(3, 8))
    if kind == "trace":
        return dict(kind=kind, scene=rng.choice(["small", "spheres"]), tris=_log(rng, 20_000, 500_000),
                    rays=_log(rng, 500, 4_000_000), bvh=rng.choice(["fp32", "q8"]), out=rng.choice(["device", "host"]))
    if kind == "adjoint":
        return dict(kind=kind, objects=rng.choice([16, 32, 64]), width=rng.randint(64, 512), height=rng.randint(64, 512),
                    spp=_log(rng, 4, 64), depth=rng.randint(3, 6))
    if kind == "batch":
        return dict(kind=kind, jobs=rng.randint(3, 12), tris=_log(rng, 10_000, 60_000), spp=rng.choice([4, 16]),
                    bvh=rng.choice(["fp32", "q8"]))
    if kind == "post":
        return dict(kind=kind, width=_log(rng, 160, 1920), height=_log(rng, 90, 1080),
                    bloom_radius=rng.choice([0.0, 0.0, 5.0, 9.0, 16.0]), tonemap=rng.choice([0, 1, 2]),
                    srgb=rng.random() < 0.7)
    return dict(kind="build", tris=_log(rng, 10_000, 500_000), rays=20_000)


# ---- scenes


@functools.lru_cache(maxsize=4)
def _geometry(scene, tris):
    """The seed-independent part of a scene."""
    if scene == "film":
        return scenes.config1(n_meshes=max(1, round(tris / 5_915)), env_w=64, env_h=32)
    return scenes.displaced_spheres(tris, 5, 640, 480, 3, env_w=64, env_h=32)


def _arrays(scene, tris, width, height, seed):
    """Scene arrays with materials, lights, environment and camera from the seed."""
    if scene == "small":
        return scenes.config0(x_res=width, y_res=height, seed=seed, n_spheres=max(1, tris // 1_280))
    base = _geometry(scene, tris)
    rng = np.random.default_rng(seed)
    mats = [dict(m, albedo=tuple(rng.uniform(0, 1, 3)), roughness=rng.uniform(0.05, 1.0),
                 metallic=float(rng.uniform() < 0.3), clearcoat=rng.uniform(0, 1), sheen=rng.uniform(0, 1))
            for m in base.materials]
    lights = (base.lights * rng.uniform(0.8, 1.2, base.lights.shape)).astype(np.float32)
    cam = dict(base.camera, x_res=width, y_res=height,
               position=(float(rng.uniform(-1, 1)), float(rng.uniform(0, 1)), -16.0))
    if scene == "film":
        env = scenes.lognormal_env(2048, 1024, seed)
    else:
        env = scenes.lognormal_env(512, 256, seed, sun=8)
    return dataclasses.replace(base, materials=mats, lights=lights, camera=cam, env=env)


def _format(case):
    return A.ER_BVH_Q8 if case.get("bvh") == "q8" else A.ER_BVH_FP32


def _film(npix, out, aov, sums):
    """Output buffers of a render: device tensors, or page-locked host tensors."""
    kw = dict(device="cuda") if out == "device" else dict(pin_memory=True)
    f = dict(beauty=torch.zeros((npix, 4), dtype=torch.float32, **kw),
             samples=torch.zeros(npix, dtype=torch.int32, **kw), pathcount=torch.zeros(npix, dtype=torch.int32, **kw))
    for k in ("normal", "tangent", "bitangent") if aov else ():
        f[k] = torch.zeros((npix, 4), dtype=torch.float32, **kw)
    if sums:
        f["sums"] = torch.zeros((npix, 3), dtype=torch.float64, **kw)
    return f


def _p(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def _batch_jobs(case, seed):
    """Views at the batch workload's resolutions, samples and depths."""
    rng = np.random.default_rng(1000 + case["jobs"])
    jobs = []
    for j in range(case["jobs"]):
        w, h = scenes.C2_RESOLUTIONS[int(rng.integers(5))]
        jobs.append(dict(scene=j, spp=int(rng.choice([case["spp"], max(1, case["spp"] // 4)])),
                         max_depth=int(rng.integers(4, 9)), seed=seed + j, width=w, height=h))
    return jobs


def _rays(arrays, n, seed):
    return scenes.random_rays(arrays, n, seed=seed)


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case, kind=kind, seed=seed)
    if kind in ("render", "noalloc"):
        arrays = _arrays(case["scene"], case["tris"], case["width"], case["height"], seed)
        st["scene"] = _lib.Scene(arrays, bvh_format=_format(case))
        flags = 0
        if kind == "render":
            flags = ((A.ER_RENDER_DEVICE_OUT if case["out"] == "device" else 0) | (A.ER_RENDER_AOV if case["aov"] else 0)
                     | (A.ER_RENDER_ENV_ALIAS if case["alias"] else 0) | (A.ER_RENDER_ACCUM_FP64 if case["fp64"] else 0))
        st["opts"] = A.er_render_opts(case["spp"], 0, case["depth"], 0, seed, flags, 0)
        st["film"] = _film(case["width"] * case["height"], case.get("out", "device"), case.get("aov", False),
                           case.get("fp64", False))
    elif kind in ("trace", "build"):
        arrays = _arrays(case.get("scene", "spheres"), case["tris"], 640, 480, seed)
        st["arrays"] = arrays
        st["rays"] = _rays(arrays, case["rays"], seed)
        if kind == "trace":
            st["scene"] = _lib.Scene(arrays, bvh_format=_format(case))
            if case["out"] == "device":
                n = case["rays"]
                st["d_rays"] = torch.from_numpy(st["rays"]).cuda()
                st["tri"] = torch.zeros(n, dtype=torch.int32, device="cuda")
                st["dist"] = torch.zeros(n, dtype=torch.float32, device="cuda")
                st["uv"] = torch.zeros((n, 2), dtype=torch.float32, device="cuda")
    elif kind == "adjoint":
        kw = dict(x_res=case["width"], y_res=case["height"], n_obj=case["objects"])
        st["scene"] = _lib.Scene(scenes.config4(param_seed=2 * seed, **kw))
        with _lib.Scene(scenes.config4(param_seed=2 * seed + 1, **kw)) as t:
            st["target"] = torch.from_numpy(t.render(4, max_depth=case["depth"], seed=seed + 7)["beauty"]).cuda()
        m, e = st["scene"].get_params()
        st["materials"] = torch.from_numpy(m).cuda().requires_grad_(True)
        st["env"] = torch.from_numpy(e).cuda().requires_grad_(True)
    elif kind == "batch":
        jobs = _batch_jobs(case, seed)
        sc = [_lib.Scene(_arrays("spheres", case["tris"], j["width"], j["height"], seed + 17 * k),
                         bvh_format=_format(case)) for k, j in enumerate(jobs)]
        st["batch"] = _lib.Batch(sc, bvh_format=_format(case))
        st["batch"].set_jobs([{k: v for k, v in j.items() if k not in ("width", "height")} for j in jobs])
        st["films"] = [_film(j["width"] * j["height"], "device", False, False) for j in jobs]
    elif kind == "post":
        g = torch.Generator(device="cuda").manual_seed(seed)
        w, h = case["width"], case["height"]
        # radiance clamped to [0, 10] as a film holds it, a fifth of it black, alpha 1
        x = torch.exp(torch.randn((h * w, 4), generator=g, device="cuda") * 1.5 - 0.5).clamp_(0.0, 10.0)
        x *= (torch.rand((h * w, 1), generator=g, device="cuda") > 0.2)
        x[:, 3] = 1.0
        st["rgba"] = x
        st["out"] = torch.zeros_like(x)
        st["ldr"] = torch.zeros((h * w, 4), dtype=torch.uint8, device="cuda")
        r = case["bloom_radius"]
        st["opts"] = A.er_post_opts(1.2, case["tonemap"], 1, int(case["srgb"]), 0, 1, 1.0, 0.3 if r else 0.0, r)
    return st


def run(st):
    L = _lib.load()
    kind, case = st["kind"], st["case"]
    if kind == "render":
        f = st["film"]
        _lib.check(L.er_render(st["scene"].h, C.byref(st["opts"]), _p(f["beauty"]), _p(f.get("normal")),
                               _p(f.get("tangent")), _p(f.get("bitangent")), _p(f["samples"]), _p(f["pathcount"]),
                               None), "er_render")
        if "sums" in f:
            _lib.check(L.er_film_read_sums(st["scene"].h, st["opts"].flags & A.ER_RENDER_DEVICE_OUT, _p(f["sums"]),
                                           None), "er_film_read_sums")
        return f
    if kind == "noalloc":
        f = st["film"]
        _lib.check(L.er_render_noalloc(st["scene"].h, C.byref(st["opts"]), _p(f["beauty"]), _p(f["samples"]),
                                       _p(f["pathcount"])), "er_render_noalloc")
        return f
    if kind == "trace":
        if case["out"] == "host":
            tri, dist, uv, _ = st["scene"].trace(st["rays"])
            return dict(tri=tri, dist=dist, uv=uv)
        _lib.check(L.er_trace_closest(st["scene"].h, _p(st["d_rays"]), case["rays"], _p(st["tri"]), _p(st["dist"]),
                                      _p(st["uv"]), A.ER_TRACE_DEVICE_PTRS, None), "er_trace_closest")
        return dict(tri=st["tri"], dist=st["dist"], uv=st["uv"])
    if kind == "adjoint":
        m, e = st["materials"], st["env"]
        m.grad = e.grad = None
        img = adjoint.render(st["scene"], m, e, case["spp"], max_depth=case["depth"], seed=st["seed"])
        loss = adjoint.l2_loss(img, st["target"])
        loss.backward()
        return dict(film=img.detach(), loss=loss.detach(), grad_materials=m.grad, grad_env=e.grad)
    if kind == "batch":
        b = st["batch"]
        b.render()
        for j, f in enumerate(st["films"]):
            _lib.check(L.er_batch_read(b.h, j, A.ER_RENDER_DEVICE_OUT, _p(f["beauty"]), _p(f["samples"]),
                                       _p(f["pathcount"])), "er_batch_read")
        return st["films"]
    if kind == "post":
        _lib.check(L.er_postprocess(_p(st["rgba"]), case["width"], case["height"], C.byref(st["opts"]), _p(st["out"]),
                                    _p(st["ldr"]), A.ER_RENDER_DEVICE_OUT), "er_postprocess")
        return dict(rgba=st["out"], ldr=st["ldr"])
    with _lib.Scene(st["arrays"], builder=A.ER_BUILDER_GPU) as s:
        tri, dist, uv, _ = s.trace(st["rays"])
    return dict(tri=tri, dist=dist, uv=uv)


# ---- what a pass cannot do without

# Per scene: vertices of a sample, tree nodes and triangles a camera or bounce ray meets on its way (counted on these
# scenes; most samples of the small ones leave at once), and the same of random rays that start among the triangles.
_PATH = {"film": (2.1, 19, 9.5), "small": (0.6, 4.5, 2.7), "spheres": (0.15, 3.6, 1.7), "diff": (0.68, 11, 5.5),
         "rays": (0, 13, 6)}


def _ray_flops(scene):
    """Four box tests (18 operations each) per node, 50 operations per triangle."""
    _, nodes, tris = _PATH[scene]
    return nodes * 4 * 18 + tris * 50


def _sample_flops(scene):
    """The camera ray; per vertex an extension ray, about 1.1 shadow rays and 900 operations of shading."""
    v = _PATH[scene][0]
    return (1 + 2.1 * v) * _ray_flops(scene) + 900 * v


def _scene_bytes(tris, env_texels):
    # 3 vertices of position, normal, uv (96 bytes) and a 128-byte node per 8 triangles; 12 bytes per texel
    return tris * (96 + 16) + env_texels * 12


def work(case):
    kind = case["kind"]
    if kind in ("render", "noalloc"):
        npix = case["width"] * case["height"]
        env = {"small": 1 << 20, "film": 2048 * 1024, "spheres": 512 * 256}[case["scene"]]
        out = 24 + (48 if case.get("aov") else 0) + (24 if case.get("fp64") else 0)
        return dict(bytes=npix * out + _scene_bytes(case["tris"], env),
                    flops=npix * case["spp"] * _sample_flops(case["scene"]))
    if kind == "trace":
        return dict(bytes=case["rays"] * (24 + 16) + _scene_bytes(case["tris"], 0),
                    flops=case["rays"] * _ray_flops("rays"))
    if kind == "adjoint":
        npix, tris = case["width"] * case["height"], case["objects"] * 1_280
        # film and its adjoint, parameters and gradients; the samples forward and once more for the gradient, whose
        # shading forms the partials too
        return dict(bytes=npix * 24 * 2 + (case["objects"] * 5 + 256 * 128 * 3) * 8 + _scene_bytes(tris, 256 * 128),
                    flops=npix * case["spp"] * (2 * _sample_flops("diff") + _PATH["diff"][0] * 1500))
    if kind == "batch":
        jobs = _batch_jobs(case, 0)
        return dict(bytes=sum(j["width"] * j["height"] * 24 + _scene_bytes(case["tris"], 512 * 256) for j in jobs),
                    flops=sum(j["width"] * j["height"] * j["spp"] * _sample_flops("spheres") for j in jobs))
    if kind == "post":
        npix = case["width"] * case["height"]
        taps = (2 * int(case["bloom_radius"] / 2) + 1) ** 2 if case["bloom_radius"] else 0
        return dict(bytes=npix * (16 + 16 + 4), flops=npix * 4 * (2 * taps + 40))
    # build: the triangles in, the leaf-ordered triangles and nodes out; sort keys, boxes and costs per triangle
    return dict(bytes=case["tris"] * (100 + 136) + case["rays"] * 40,
                flops=case["tris"] * 2_000 + case["rays"] * _ray_flops("rays"))


# ---- results in 64 bits

def _brute_force(arrays, rays):
    """Closest hit of each ray over every triangle: the hit with the smallest |position - origin|, the position being
    the smooth-shading one where the surface is locally convex."""
    P, N = (torch.from_numpy(np.asarray(a, np.float64)).cuda() for a in (arrays.positions, arrays.normals))
    R = torch.from_numpy(rays.astype(np.float64)).cuda()
    R[:, 3:] /= R[:, 3:].norm(dim=1, keepdim=True)
    v0, e1, e2 = P[:, 0], P[:, 1] - P[:, 0], P[:, 2] - P[:, 0]
    dist = torch.zeros(len(R), dtype=torch.float64, device="cuda")
    uv = torch.zeros((len(R), 2), dtype=torch.float64, device="cuda")
    step = max(1, 8_000_000 // max(1, len(P)))
    for a in range(0, len(R), step):
        o, d = R[a:a + step, None, :3], R[a:a + step, None, 3:]
        p = torch.linalg.cross(d.expand(-1, len(P), -1), e2[None])
        det = (e1[None] * p).sum(-1)
        tv = o - v0[None]
        u = (tv * p).sum(-1) / det
        q = torch.linalg.cross(tv, e1[None].expand_as(tv))
        v = (d * q).sum(-1) / det
        t = (e2[None] * q).sum(-1) / det
        ok = (det.abs() >= 1e-7) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t >= 0)
        i, k = ok.nonzero(as_tuple=True)
        uu, vv, tt = u[i, k, None], v[i, k, None], t[i, k, None]
        oo, dd, n = R[a + i, :3], R[a + i, 3:], N[k]
        g = oo + dd * tt
        pr = [g - n[:, c] * ((g - P[k, c]) * n[:, c]).sum(-1, keepdim=True) for c in range(3)]
        sp = pr[0] + (pr[1] - pr[0]) * uu + (pr[2] - pr[0]) * vv
        sn = n[:, 0] + (n[:, 1] - n[:, 0]) * uu + (n[:, 2] - n[:, 0]) * vv
        pos = torch.where(((sp - g) * sn).sum(-1, keepdim=True) > 0, sp, g)
        w = torch.full_like(t, math.inf)
        w[i, k] = (pos - oo).norm(dim=1)
        best, at = w.min(dim=1)
        hit = torch.isfinite(best)
        row = torch.arange(len(at), device="cuda")
        dist[a:a + step] = torch.where(hit, best, 0.0)
        uv[a:a + step] = torch.where(hit[:, None], torch.stack([u[row, at], v[row, at]], 1), 0.0)
    return dist, uv


def exact(case, seed):
    if case["kind"] in ("trace", "build"):
        if case["tris"] * case["rays"] > 4e8:  # brute force over every pair: too long beyond this
            return None
        arrays = _arrays(case.get("scene", "spheres"), case["tris"], 640, 480, seed)
        dist, uv = _brute_force(arrays, _rays(arrays, case["rays"], seed))
        return dict(tri=None, dist=dist, uv=uv)
    if case["kind"] == "post":
        st = prepare(case, seed)
        w, h, o = case["width"], case["height"], st["opts"]
        x = st["rgba"].double() * float(o.exposure)
        b = int(o.bloom_radius / 2) if o.bloom_power else 0
        if b > 0:
            c = torch.arange(-b, b + 1, dtype=torch.float64, device="cuda")
            sd = float(o.bloom_radius)
            k = torch.exp(-(c[:, None] ** 2 + c[None] ** 2) / (2 * sd * sd)) / (2 * math.pi * sd * sd)
            bright = torch.where(x[:, :3].mean(1, keepdim=True) < float(o.bloom_threshold), 0.0, x)
            img = bright.view(h, w, 4).permute(2, 0, 1)[:, None]
            blur = torch.zeros_like(img)
            if h > 2 * b and w > 2 * b:
                blur[:, :, b:h - b, b:w - b] = torch.nn.functional.conv2d(img, k[None, None])
            x = x + blur[:, 0].permute(1, 2, 0).reshape(-1, 4) * float(o.bloom_power)
        if o.tonemap == A.ER_TONEMAP_REINHARD:
            x = x / (1 + x)
        elif o.tonemap == A.ER_TONEMAP_ACES:
            y = x * 0.6
            x = (y * (2.51 * y + 0.03) / (y * (2.43 * y + 0.59) + 0.14)).clamp(0, 1)
        x = x.clamp(0, 1)
        if o.srgb:
            x = x ** (1 / 2.2)
        return dict(rgba=x.view(h, w, 4).flip(0).reshape(-1, 4), ldr=None)
    # films and gradients: a Monte Carlo path is another path as soon as one of its hits, texels or lobes is decided by
    # the last bit of a 32-bit number, so a 64-bit path tracer gives the same film only in the limit of many samples
    return None
