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
