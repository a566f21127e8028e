"""Renders that count their traversal (profile bit 1) over a pass with a NaN path, which visits no
node, as in the renders that do not count."""
import numpy as np
import pytest

import gianduia_b200 as G
from gianduia_b200 import scenes

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(120)]


def test_counting_render_with_a_nan_path(tmp_path):
    ctx = G.GpuContext(0)
    sid = ctx.upload(G.HostScene.load_xml(scenes.microfacet(str(tmp_path / "mf"))))
    film, st = ctx.render(sid, spp=8, first_pass=168, max_depth=16, batched=True, profile=2)
    ref, _ = ctx.render(sid, spp=8, first_pass=168, max_depth=16, batched=True)
    assert st["paths"] == 8 * 1024 * 1024 and st["extend_nodes"] > st["extend_rays"]
    assert np.array_equal(film[..., :4], ref[..., :4])
    ctx.close()


def test_counting_render_counts_the_lanes_that_work(tmp_path):
    """A triangle pass shares the leaves of all lanes out over the warp: its busy lanes are the
    triangles it tests, up to four of each leaf, and instances are entered in steps of their own."""
    ctx = G.GpuContext(0)
    sid = ctx.upload(G.HostScene.load_xml(scenes.microfacet(str(tmp_path / "mf"), width=128, height=128, grid=16)))
    counts = []
    for leaf_batch in (32, 16, 4):
        ctx.set_tune(sid, leaf_batch=leaf_batch)
        film, st = ctx.render(sid, spp=4, max_depth=8, batched=True, profile=2)
        tris, ls, lw = st["extend_tris"], st["extend_leaf_steps"], st["extend_leaf_warp_steps"]
        assert 0 < tris < ls <= 32 * lw
        assert 0 < st["extend_node_warp_steps"] <= st["extend_nodes"] <= 32 * st["extend_node_warp_steps"]
        # a ray's visits do not depend on the schedule
        counts.append((st["extend_nodes"], tris, ls))
    assert counts[0] == counts[1] == counts[2]
    ctx.close()
