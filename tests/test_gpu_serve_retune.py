"""The serving settings and the pool change between jobs that follow each other at once (a round of
the job before is then still queued), and a context closes right after its last job."""
import numpy as np
import pytest

import gianduia_b200 as G
from gianduia_b200 import scenes

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(120)]


@pytest.mark.parametrize("graphs", [1, 0])
def test_settings_change_behind_a_queued_round(tmp_path, graphs):
    hs = G.HostScene.load_xml(scenes.cornell(str(tmp_path), width=48, height=48, spp=3))
    ref = None
    for _ in range(3):
        ctx = G.GpuContext(0)
        sid = ctx.upload(hs)
        for pool, iters in ((16, 4), (17, 64), (18, 2), (18, 4), (19, 8)):
            ctx.serve_tune(pool_log2=pool, round_iters=iters, graphs=graphs)
            film, st = ctx.wait(ctx.submit(sid, spp=3, max_depth=6), timeout_ms=20000)
            assert st["state"] == "done"
            ref = film if ref is None else ref
            assert np.array_equal(film[..., :4], ref[..., :4])
            film, _ = ctx.render(sid, spp=3, max_depth=6)
            assert np.array_equal(film[..., :4], ref[..., :4])
        ctx.close()
