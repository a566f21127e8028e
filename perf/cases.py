"""Timed cases over the framework's public entry points (gianduia_b200): ray batches, renders,
served jobs, mesh refits and post-processing, from the smallest calls to the largest.

A case is a dict of plain values. prepare() makes what a program has in hand before the
call -- a resident scene, its rays, new vertex positions, an image -- from the seed alone;
run() is one call (or the few calls that belong together) as a program makes it. Scene
geometry of the XML scenes is fixed by the generators in gianduia_b200.scenes; the seed
picks the first of the sample passes that are rendered, so another seed renders other samples.
"""
import math
import os
import tempfile

import numpy as np
import torch

import gianduia_b200 as G
from gianduia_b200 import scenes, serving

SCENE_DIR = os.path.join(tempfile.gettempdir(), "gianduia_perf_scenes_%d" % os.getuid())
THIN_LENS = {"lens_radius": 0.05, "focal_distance": 3.5, "blades": 6, "k1": 0.02, "vignetting": True}
FIRST_PASSES = 104   # a render starts at one of the first sample passes
TONEMAPPERS = ("linear", "reinhard", "uncharted2", "aces", "khronos_pbr", "agx", "agx_punchy")


def listed():
    return [
        # a handful of rays on a small mesh: picking, autofocus, light probes
        dict(name="rays_probe", kind="rays", tris=4096, rays=1000, query="closest", buffers="device", tmax="inf", tree="host"),
        # a caller's own batch in host memory, copied in and out by the call
        dict(name="rays_host_batch", kind="rays", tris=65537, rays=65539, query="closest", buffers="host", tmax="inf", tree="host"),
        # bounded visibility segments (baking, ambient occlusion) on a mesh tree built at upload
        dict(name="rays_any_segments", kind="rays", tris=300007, rays=3000017, query="any", buffers="device", tmax="segment", tree="device"),
        # the traversal micro-benchmark at its full size
        dict(name="rays_closest_16m", kind="rays", tris=1 << 20, rays=1 << 24, query="closest", buffers="device", tmax="inf", tree="host"),
        # an interactive preview: few samples of a small image, the reference's default film filter
        dict(name="render_preview", kind="render", scene="cornell", width=333, height=211, spp=4, depth=8, batched=True, filter="default"),
        # the drop-in integrator as the host framework calls it: one pass after another
        dict(name="render_cornell_plain", kind="render", scene="cornell", width=256, height=256, spp=16, depth=8, batched=False, filter="box"),
        # volpath: homogeneous media, index boundaries, transmittance queries
        dict(name="render_volumetric", kind="render", scene="volumetric", width=512, height=512, spp=16, depth=32, batched=True, filter="box"),
        # textures, normal and bump maps through a thin lens
        dict(name="render_textured_lens", kind="render", scene="textures", width=640, height=360, spp=16, depth=8, batched=True, filter="box"),
        # the headline render: 5.2M triangles, rough materials, 67M paths
        dict(name="render_microfacet", kind="render", scene="microfacet", grid=64, width=1024, height=1024, spp=64, depth=16, batched=True, filter="box"),
        # a burst of requests on the job server, their films collected as they finish
        dict(name="serve_mix", kind="serve", jobs=12, mix=4, grid=24, res=512, spp=16),
        # one frame of an animation: new vertex positions for a resident mesh, then its rays
        dict(name="refit_frame", kind="refit", tris=300007, rays=500009),
        # the finished image through bloom, the tone curve and 8-bit conversion
        dict(name="post_image", kind="post", width=1024, height=1024, tonemapper="agx", bloom=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("rays", "rays", "rays", "render", "render", "render", "render", "serve", "refit", "post"))
    if kind == "rays":
        host = rng.random() < 0.25
        return dict(kind="rays", tris=_log_int(rng, 3000, 1 << 20), rays=_log_int(rng, 500, (1 << 18) if host else (1 << 23)),
                    query=rng.choice(("closest", "any")), buffers="host" if host else "device",
                    tmax=rng.choice(("inf", "segment")), tree=rng.choice(("host", "device")))
    if kind == "render":
        scene = rng.choice(("cornell", "volumetric", "microfacet", "textures"))
        batched = rng.random() < 0.7
        spp = _log_int(rng, 1, 32)
        w, h = _log_int(rng, 100, 1024), _log_int(rng, 100, 1024)
        most = {"cornell": 8e6, "volumetric": 4e6, "microfacet": 16e6, "textures": 4e6}[scene] / (1 if batched else 4)
        spp = max(1, min(spp, int(most / (w * h))))
        filt = rng.choice(("box", "default")) if scene in ("cornell", "volumetric") else "box"
        c = dict(kind="render", scene=scene, width=w, height=h, spp=spp, depth=rng.randint(8, 32), batched=batched, filter=filt)
        return dict(c, grid=rng.choice((12, 16, 24))) if scene == "microfacet" else c
    if kind == "serve":
        return dict(kind="serve", jobs=rng.randint(2, 12), mix=rng.randint(5, 10000), grid=24, res=rng.choice((128, 256, 512)), spp=rng.choice((4, 16)))
    if kind == "refit":
        return dict(kind="refit", tris=_log_int(rng, 5000, 600000), rays=_log_int(rng, 10000, 1000000))
    return dict(kind="post", width=_log_int(rng, 200, 2048), height=_log_int(rng, 200, 2048),
                tonemapper=rng.choice(TONEMAPPERS), bloom=rng.random() < 0.7)


# ---------------------------------------------------------------- what a program keeps
_contexts = {}


def _context(use):
    """One context per use, as a program keeps it: the renderer's, and the job server's."""
    if use not in _contexts:
        _contexts[use] = G.GpuContext(0)
    return _contexts[use]


class _Resident:
    """A scene in device memory, freed with the state that holds it."""

    def __init__(self, ctx, host):
        self.ctx = ctx
        self.id = ctx.upload(host)

    def __del__(self):
        try:
            self.ctx.free_scene(self.id)
        except Exception:
            pass


def _scene_file(scene, width, height, spp, depth, filt, grid=24):
    d = os.path.join(SCENE_DIR, "%s_%d_%d_%d_%d_%s" % (scene, width, height, spp, depth, filt))
    if scene == "cornell":
        return scenes.cornell(d, width=width, height=height, spp=spp, max_depth=depth, filter=filt)
    if scene == "volumetric":
        return scenes.volumetric(d, width=width, height=height, spp=spp, max_depth=depth, filter=filt)
    if scene == "textures":
        return scenes.textures(d, width=width, height=height, spp=spp, max_depth=depth, lens=THIN_LENS, maps=True)
    # the sphere grid's mesh files (4,096 of them at grid 64) are written once; film size,
    # samples and depth are given with the call
    return scenes.microfacet(os.path.join(SCENE_DIR, "microfacet_%d" % grid), grid=grid)


def _soup(tris, seed):
    return scenes.random_triangles(tris, seed=seed)


def _rays(n, tmax, seed):
    """Origins uniform in [-0.5, 1.5]^3, directions uniform on the sphere, as [n, 8] on the
    GPU; "segment": lengths uniform in [0.05, 1]."""
    g = torch.Generator(device="cuda").manual_seed(seed + 77)
    r = torch.empty((n, 8), dtype=torch.float32, device="cuda")
    r[:, 0:3] = torch.rand((n, 3), device="cuda", generator=g) * 2.0 - 0.5
    r[:, 3] = 1e-4
    d = torch.randn((n, 3), device="cuda", generator=g)
    r[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    r[:, 7] = math.inf if tmax == "inf" else torch.rand((n,), device="cuda", generator=g) * 0.95 + 0.05
    return r


def _deformed(tris, seed):
    """The next frame's positions: the soup sheared and bent by a smooth field."""
    p = tris.reshape(-1, 3)
    phase = float(np.random.default_rng(seed + 9).uniform(0.0, 6.28))
    q = p + 0.03 * np.sin(5.0 * p[:, [1, 2, 0]] + phase)
    return np.ascontiguousarray(q, np.float32).reshape(-1, 9)


def _requests(case):
    out = []
    for r in serving.make_requests(case["jobs"], seed=case["mix"]):
        out.append(dict(r, res=min(r["res"], case["res"]), spp=min(r["spp"], case["spp"])))
    return out


def prepare(case, seed):
    kind = case["kind"]
    ctx = _context("serve" if kind == "serve" else "render")
    if kind == "rays":
        host = G.HostScene.from_triangles(_soup(case["tris"], seed), device_blas=case["tree"] == "device")
        rays = _rays(case["rays"], case["tmax"], seed)
        s = dict(kind=kind, query=case["query"], buffers=case["buffers"], ctx=ctx, scene=_Resident(ctx, host), n=case["rays"])
        if case["buffers"] == "host":
            s["rays"] = rays.cpu().numpy()
        else:
            s["rays"] = rays
            s["out"] = torch.empty((case["rays"], 5), dtype=torch.float32, device="cuda") if case["query"] == "closest" \
                else torch.empty((case["rays"],), dtype=torch.uint8, device="cuda")
        return s
    if kind == "render":
        host = G.HostScene.load_xml(_scene_file(case["scene"], case["width"], case["height"], case["spp"], case["depth"], case["filter"],
                                                    case.get("grid", 0)))
        return dict(kind=kind, ctx=ctx, scene=_Resident(ctx, host), spp=case["spp"], first=seed % FIRST_PASSES,
                    batched=case["batched"], depth=case["depth"], width=case["width"], height=case["height"])
    if kind == "serve":
        ids = {n: _Resident(ctx, G.HostScene.load_xml(_scene_file(n, 256, 256, 16, 16, "box", case["grid"])))
               for n in serving.SCENES}
        return dict(kind=kind, ctx=ctx, scenes=ids, jobs=_requests(case), first=seed % FIRST_PASSES)
    if kind == "refit":
        t = _soup(case["tris"], seed)
        return dict(kind=kind, ctx=ctx, scene=_Resident(ctx, G.HostScene.from_triangles(t)), positions=_deformed(t, seed), n=case["rays"],
                    rays=_rays(case["rays"], "inf", seed), out=torch.empty((case["rays"], 5), dtype=torch.float32, device="cuda"))
    # a linear image with the range of a render: a smooth base, highlights far above 1
    rng = np.random.default_rng(seed)
    h, w = case["height"], case["width"]
    img = rng.gamma(1.5, 0.4, size=(h, w, 3)).astype(np.float32)
    img[rng.random((h, w)) < 0.002] *= np.float32(40.0)
    return dict(kind=kind, ctx=ctx, image=img, tonemapper=case["tonemapper"], bloom=case["bloom"])


def _hits(out):
    return {"t": out[:, 0], "u": out[:, 1], "v": out[:, 2], "inst": out.view(torch.int32)[:, 3], "prim": out.view(torch.int32)[:, 4]}


def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "rays":
        if s["buffers"] == "host":
            if s["query"] == "any":
                return ctx.trace_any(s["scene"].id, s["rays"])
            h = ctx.trace_closest(s["scene"].id, s["rays"])
            return {k: h[k] for k in ("t", "u", "v", "inst", "prim")}
        if s["query"] == "any":
            ctx.trace_any_dev(s["scene"].id, s["rays"].data_ptr(), s["n"], s["out"].data_ptr())
            return s["out"]
        ctx.trace_closest_dev(s["scene"].id, s["rays"].data_ptr(), s["n"], s["out"].data_ptr())
        return _hits(s["out"])
    if kind == "render":
        film, _ = ctx.render(s["scene"].id, spp=s["spp"], first_pass=s["first"], max_depth=s["depth"], batched=s["batched"],
                             width=s["width"], height=s["height"])
        return film
    if kind == "serve":
        jobs = [ctx.submit(s["scenes"][r["scene"]].id, width=r["res"], height=r["res"], spp=r["spp"], max_depth=r["max_depth"],
                           integrator=1 if r["scene"] == "volumetric" else 0, first_pass=s["first"]) for r in s["jobs"]]
        return [ctx.wait(j)[0] for j in jobs]
    if kind == "refit":
        ctx.refit_mesh(s["scene"].id, 0, s["positions"])
        ctx.trace_closest_dev(s["scene"].id, s["rays"].data_ptr(), s["n"], s["out"].data_ptr())
        return _hits(s["out"])
    hdr, rgb8 = ctx.post(s["image"], tonemapper=s["tonemapper"], bloom=s["bloom"])
    return {"hdr": hdr, "rgb8": rgb8}


# ---------------------------------------------------------------- work
def _scene_tris(scene, grid):
    return grid * grid * 1280 + 2 if scene == "microfacet" else {"cornell": 36, "volumetric": 48, "textures": 60}[scene]


def _ray_flops(tris):
    """One ray: four child boxes (6 planes, 2 operations each, and the interval) on every
    level of a 4-wide tree, and one triangle."""
    return (math.log(max(tris, 4), 4) + 1.0) * 4 * 14 + 50


def _scene_bytes(tris):
    return tris * (48 + 64 + 128 / 3.0)   # triangles, attributes, about a node per three triangles


def work(case):
    kind = case["kind"]
    if kind == "rays":
        out = 20 if case["query"] == "closest" else 1
        return {"bytes": case["rays"] * (32 + out) + case["tris"] * (48 + 128 / 3.0), "flops": case["rays"] * _ray_flops(case["tris"])}
    if kind in ("render", "serve"):
        grid = case.get("grid", 0)
        jobs = [dict(scene=case["scene"], paths=case["width"] * case["height"] * case["spp"], film=case["width"] * case["height"])] \
            if kind == "render" else [dict(scene=r["scene"], paths=r["res"] ** 2 * r["spp"], film=r["res"] ** 2) for r in _requests(case)]
        b = sum(_scene_bytes(_scene_tris(n, grid)) for n in {j["scene"] for j in jobs}) + sum(28 * j["film"] for j in jobs)
        # about three bounces a path (six with media), each a closest hit, a shadow query and 300 operations of shading
        f = sum(j["paths"] * (6 if j["scene"] == "volumetric" else 3) * (2 * _ray_flops(_scene_tris(j["scene"], grid)) + 300) for j in jobs)
        return {"bytes": b, "flops": f}
    if kind == "refit":
        t = case["tris"]
        return {"bytes": t * (36 + 48 + 128 / 3.0) + case["rays"] * 52, "flops": t * 30 + case["rays"] * _ray_flops(t)}
    px = case["width"] * case["height"]
    return {"bytes": px * (12 + 12 + 3), "flops": px * (250 if case["bloom"] else 60)}


# ---------------------------------------------------------------- 64-bit values
def _closest64(tris, rays):
    """Closest hit of every ray by testing every triangle (Moller-Trumbore) in 64 bits:
    distance and barycentric coordinates, inf and 0 on a miss."""
    v0, v1, v2 = (torch.from_numpy(tris[:, k].astype(np.float64)).cuda() for k in range(3))
    e1, e2 = v1 - v0, v2 - v0
    best = torch.full((rays.shape[0],), math.inf, dtype=torch.float64, device="cuda")
    bu, bv = torch.zeros_like(best), torch.zeros_like(best)
    step = max(1, (1 << 24) // tris.shape[0])

    def dot(a, b):
        return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]

    def cross(a, b):
        return (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0])

    for k in range(0, rays.shape[0], step):
        r = rays[k:k + step].double()
        o = [r[:, a, None] for a in range(3)]
        d = [r[:, 4 + a, None] for a in range(3)]
        E1, E2, V0 = ([x[None, :, a] for a in range(3)] for x in (e1, e2, v0))
        p = cross(d, E2)
        det = dot(E1, p)
        tv = [o[a] - V0[a] for a in range(3)]
        u = dot(tv, p) / det
        q = cross(tv, E1)
        v = dot(d, q) / det
        t = dot(E2, q) / det
        ok = (det.abs() > 1e-8) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t > r[:, 3, None]) & (t < r[:, 7, None])
        t = torch.where(ok, t, math.inf)
        m, i = t.min(dim=1)
        hit = torch.isfinite(m)
        row = torch.arange(r.shape[0], device="cuda")
        best[k:k + step] = m
        bu[k:k + step] = torch.where(hit, u[row, i], 0.0)
        bv[k:k + step] = torch.where(hit, v[row, i], 0.0)
    return best, bu, bv


def exact(case, seed):
    """Distances and barycentrics of ray batches small enough to test every triangle. The
    renders have no closed form; the bloom pyramid is defined in half precision."""
    if case["kind"] == "rays" and case["query"] == "closest" and case["rays"] * case["tris"] <= 5e9:
        t, u, v = _closest64(_soup(case["tris"], seed), _rays(case["rays"], case["tmax"], seed))
        return {"t": t, "u": u, "v": v, "inst": None, "prim": None}
    if case["kind"] == "post" and not case["bloom"] and case["tonemapper"] in ("linear", "reinhard"):
        x = prepare(dict(case), seed)["image"].astype(np.float64)
        y = x @ np.array([0.2126, 0.7152, 0.0722])   # reinhard: the luminance is mapped, the hue kept
        s = 1.0 if case["tonemapper"] == "linear" else ((y / (1.0 + y)) / np.maximum(y, 1e-5))[..., None]
        return {"hdr": x * s, "rgb8": None}
    return None
