"""Ray batches around the sizes from which rays go 32 to a warp instead of a few to each warp of the
full grid (4 rays a warp in small trees, 8 in larger ones), against the oracle."""
import numpy as np
import pytest

import gianduia_b200 as G
from gianduia_b200 import scenes
from oracle import pyoracle as O

from test_gpu_traversal import compare_closest

pytestmark = pytest.mark.gpu

WARPS = 148 * 8 * 4


@pytest.mark.parametrize("tris,per_warp", [(500, 4), (30000, 8)])
@pytest.mark.parametrize("extra", [-1, 0, 1, 130])
def test_batches_around_the_line(tris, per_warp, extra):
    tri = scenes.random_triangles(tris, seed=4)
    hs = G.HostScene.from_triangles(tri)
    assert (hs.desc.num_nodes >= 4096) == (per_warp == 8)
    n = WARPS * per_warp + extra
    rays = scenes.random_rays(n, seed=n)
    ctx = G.GpuContext(0)
    sid = ctx.upload(hs)
    osc = O.Scene.from_triangles(tri)
    ref = osc.trace(rays)
    compare_closest(ctx.trace_closest(sid, rays), ref, rays, "%d rays" % n)
    assert np.array_equal(ctx.trace_any(sid, rays), osc.trace(rays, anyhit=True)[0])
    ctx.set_tune(sid, trace_blocks=3)
    compare_closest(ctx.trace_closest(sid, rays), ref, rays, "%d rays, 3 blocks" % n)
    ctx.close()
