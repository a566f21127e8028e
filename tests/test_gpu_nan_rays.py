"""Rays with a NaN in their origin or direction (degenerate BSDF samples) hit no triangle and
no sphere, and a cube only at a finite tMax: the oracle's hits, without a walk through the
whole scene. The slow test renders the sample pass of the sphere grid whose path of that kind
ran into the traversal's iteration limit."""
import numpy as np
import pytest

import gianduia_b200 as G
from gianduia_b200 import scenes
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

SHAPES = """<scene>
<camera type="perspective"><transform name="toWorld"><lookat origin="0,0,6" target="0,0,0" up="0,1,0"/></transform></camera>
<sampler type="independent"/><integrator type="path_gpu"/>
<primitive><transform name="toWorld"><scale value="1.5"/><rotate axis="1 1 0" angle="30"/><translate x="-1" y="0" z="0"/></transform>
<shape type="sphere"><float name="radius" value="0.7"/></shape></primitive>
%s</scene>"""
CUBE = """<primitive><transform name="toWorld"><rotate axis="0 1 1" angle="40"/><translate x="1.2" y="0.3" z="-0.5"/></transform>
<shape type="cube"><vector name="extents" value="0.5, 0.8, 0.3"/></shape>
<emitter type="area"><color name="radiance" value="1 1 1"/></emitter></primitive>"""


@pytest.fixture(scope="module")
def ctx():
    c = G.GpuContext(0)
    yield c
    c.close()


def _nan_rays():
    r = scenes.random_rays(4096, seed=9)
    rng = np.random.default_rng(10)
    r[:2048, 7] = rng.uniform(0.1, 3.0, 2048).astype(np.float32)   # finite tMax for half of them
    bad = rng.random((4096, 3)) < 0.4
    which = rng.integers(0, 3, 4096)                               # origin, direction, both
    for c in range(3):
        r[bad[:, c] & (which != 1), c] = np.nan
        r[bad[:, c] & (which != 0), 4 + c] = np.nan
    return r


@pytest.mark.parametrize("scene", ["soup", "sphere", "cube"])
def test_nan_rays_match_the_oracle(ctx, tmp_path, scene):
    rays = _nan_rays()
    if scene == "soup":
        tri = scenes.random_triangles(2000, seed=8)
        hs, osc = G.HostScene.from_triangles(tri), O.Scene.from_triangles(tri)
    else:
        xml = str(tmp_path / "s.xml")
        with open(xml, "w") as f:
            f.write(SHAPES % (CUBE if scene == "cube" else ""))
        hs, osc = G.HostScene.load_xml(xml), O.Scene.load(xml)
    sid = ctx.upload(hs)
    g, ref = ctx.trace_closest(sid, rays), osc.trace(rays)
    for k in ("inst", "prim"):
        assert np.array_equal(g[k], ref[k]), k
    assert np.array_equal(g["t"], ref["t"])
    # any hit: the oracle's answer for segments; an unbounded ray is occluded when it has a
    # closest hit (the reference's any-hit query also takes a cube's "hit" at infinity)
    occ, bounded = ctx.trace_any(sid, rays), np.isfinite(rays[:, 7])
    assert np.array_equal(occ[bounded], osc.trace(rays, anyhit=True)[0][bounded])
    assert np.array_equal(occ[~bounded], g["inst"][~bounded] >= 0)
    ctx.free_scene(sid)


def test_render_with_a_nan_path(ctx, tmp_path):
    hs = G.HostScene.load_xml(scenes.microfacet(str(tmp_path / "mf")))
    sid = ctx.upload(hs)
    _, st = ctx.render(sid, spp=8, first_pass=168, max_depth=16, batched=True)
    assert st["paths"] == 8 * 1024 * 1024
    ctx.free_scene(sid)
