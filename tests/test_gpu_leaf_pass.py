"""The warp's shared leaf pass and the spreading of small batches: leaves of 1 to 16 triangles
(triangles around one centroid stay together in a leaf; more become several leaves) and
batches around the sizes where rays start to share a warp, against the oracle. Triangles
around one centroid are scaled copies in parallel planes, so every ray that hits a cluster has
up to its full count of candidates in one leaf."""
import numpy as np
import pytest

import gianduia_b200 as G
from oracle import pyoracle as O

from test_gpu_traversal import compare_closest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = G.GpuContext(0)
    yield c
    c.close()


def _clusters(count, per, seed):
    """count clusters of `per` triangles whose bounding boxes share one centre."""
    rng = np.random.default_rng(seed)
    centre = rng.integers(0, 64, (count, 1, 1, 3)) / 64.0          # exact in float32: equal centroids
    half = rng.integers(1, 64, (count, per, 1, 3)) / 1024.0
    corner = np.array([[-1, -1, 1], [1, -1, -1], [-1, 1, -1]], np.float64)
    return (centre + half * corner).reshape(-1, 3, 3).astype(np.float32)


def _rays(n, seed):
    rng = np.random.default_rng(seed)
    o = rng.uniform(-0.5, 1.5, (n, 3))
    to = rng.uniform(0.0, 1.0, (n, 3))
    d = to - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([o, np.full((n, 1), 1e-4), d, np.full((n, 1), np.inf)], axis=1).astype(np.float32)


@pytest.mark.parametrize("per", [1, 3, 4, 5, 15, 16, 17, 40])
def test_leaf_sizes(ctx, per):
    tri = _clusters(400, per, per)
    rays = _rays(20000, per)
    sid = ctx.upload(G.HostScene.from_triangles(tri))
    osc = O.Scene.from_triangles(tri)
    # clusters drawn on one centre can hold equal triangles: those are ties
    st = compare_closest(ctx.trace_closest(sid, rays), osc.trace(rays), rays, "clusters of %d" % per, max_tie_frac=0.05)
    assert st["hits"] > 1000
    assert np.array_equal(ctx.trace_any(sid, rays), osc.trace(rays, anyhit=True)[0])
    ctx.free_scene(sid)


@pytest.mark.parametrize("n", [1, 2, 31, 33, 591, 593, 4735, 4737, 9473, 151551, 151553])
def test_batch_sizes(ctx, n):
    tri = _clusters(300, 3, 5)
    rays = _rays(n, n)
    sid = ctx.upload(G.HostScene.from_triangles(tri))
    osc = O.Scene.from_triangles(tri)
    compare_closest(ctx.trace_closest(sid, rays), osc.trace(rays), rays, "%d rays" % n, max_tie_frac=0.05)
    assert np.array_equal(ctx.trace_any(sid, rays), osc.trace(rays, anyhit=True)[0])
    ctx.free_scene(sid)
