"""Non-finite refit positions are refused and change nothing, at the sizes around which the check
moves from the host to the device (256 KB of positions)."""
import numpy as np
import pytest

import gianduia_b200 as G
from gianduia_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 7281, 7282, 40001])
def test_refit_positions_must_be_finite(n):
    ctx = G.GpuContext(0)
    tri = scenes.random_triangles(n, seed=6).reshape(-1, 9)
    sid = ctx.upload(G.HostScene.from_triangles(tri))
    rays = scenes.random_rays(20000, seed=7)
    before = ctx.trace_closest(sid, rays)
    for value in (np.nan, np.inf, -np.inf):
        for at in (0, n * 9 - 1, n * 9 // 2):
            bad = tri.copy()
            bad.reshape(-1)[at] = value
            with pytest.raises(G.GndError) as e:
                ctx.refit_mesh(sid, 0, bad)
            assert e.value.status == G.GND_ERR_INVALID
    assert ctx.trace_closest(sid, rays).tobytes() == before.tobytes()
    ctx.refit_mesh(sid, 0, tri)
    assert ctx.trace_closest(sid, rays).tobytes() == before.tobytes()
    ctx.close()
