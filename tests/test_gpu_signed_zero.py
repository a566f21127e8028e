"""Axis-parallel rays whose zero components are negative zeros, with their origin on a box plane of
the mesh: an instance's transform turns -0 into +0, the reciprocal changes its sign with it, and
a box whose lo plane holds the origin is entered or not accordingly. The remaining component is
denormal, so its reciprocal is infinite as well and every plane of the slab test lies at
infinity or is NaN: the only case in which that sign decides. Hits equal the oracle's."""
import itertools

import numpy as np
import pytest

import gianduia_b200 as G
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def _mesh(side):
    """Eight huge triangles whose box begins (side 1) or ends (side -1) at x = 0, eight more far away."""
    tri = []
    for k in range(8):
        z = 0.02 + 0.03 * k
        tri.append([[0, -1e18, z], [0, 1e18, z], [side * 1e18, 0, z]])
        z = -1.0 + 0.25 * k
        tri.append([[-side * 3e18, -1e18, z], [-side * 3e18, 1e18, z], [-side * 2e18, 0, z]])
    return np.array(tri, np.float32)


def _rays():
    rays = []
    for dx, dy, dz, oy, oz in itertools.product((0.0, -0.0), (0.0, -0.0), (1e-39, 3e-39), (0.0, 3e17, -1e17), (0.0, -0.05)):
        rays.append([0.0, oy, oz, 1e-4, dx, dy, dz, np.inf])
    return np.array(rays, np.float32)


@pytest.mark.parametrize("side", [1, -1])
def test_negative_zero_directions(side):
    tri, rays = _mesh(side), _rays()
    assert np.signbit(rays[:, 4]).any() and (rays[:, 6] > 0).all()
    ctx = G.GpuContext(0)
    sid = ctx.upload(G.HostScene.from_triangles(tri))
    osc = O.Scene.from_triangles(tri)
    ref, got = osc.trace(rays), ctx.trace_closest(sid, rays)
    assert np.array_equal(got["inst"], ref["inst"])
    assert np.array_equal(got["prim"], ref["prim"]) and np.array_equal(got["t"], ref["t"])
    assert np.array_equal(ctx.trace_any(sid, rays), osc.trace(rays, anyhit=True)[0])
    if side > 0:
        assert (ref["inst"] >= 0).any()   # entered through +inf
    ctx.close()
