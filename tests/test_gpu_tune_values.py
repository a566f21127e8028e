"""Settings that select code of their own render the defaults' film sums, and the autotuner tells
apart only settings that run different code."""
import numpy as np
import pytest

import gianduia_b200 as G
from gianduia_b200 import scenes

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(300)]


@pytest.fixture(scope="module")
def setup(tmp_path_factory):
    d = tmp_path_factory.mktemp("tune")
    ctx = G.GpuContext(0)
    grid = ctx.upload(G.HostScene.load_xml(scenes.microfacet(str(d / "g"), width=64, height=48, spp=8, max_depth=8, grid=24, seed=3)))
    yield ctx, grid
    ctx.close()


def test_distinct_settings(setup):
    ctx, sid = setup
    base, _ = ctx.render(sid, batched=True)
    default = ctx.get_tune(sid)
    for v in (dict(leaf_batch=1), dict(leaf_batch=4), dict(leaf_batch=15), dict(shadow_leaf_batch=1), dict(shadow_leaf_batch=8),
              dict(stack_smem=16, leaf_batch=2), dict(stack_smem=16, shadow_leaf_batch=4, trav_blocks=1)):
        ctx.set_tune(sid, **v)
        film, _ = ctx.render(sid, batched=True)
        assert np.array_equal(film[..., :4], base[..., :4]), v
        ctx.set_tune(sid, **default)


def test_autotune_leaves_equal_settings_alone(setup):
    ctx, sid = setup
    default = ctx.get_tune(sid)
    ctx.set_tune(sid, leaf_batch=24, shadow_leaf_batch=20)   # both are taken as 16, as every value above
    tune, _ = ctx.autotune(sid, spp=2, budget_ms=4000)
    assert tune["leaf_batch"] in (24, 32, 8) and tune["shadow_leaf_batch"] in (20, 32, 8)
    # 32 only by way of 8: never in place of the value that runs the same code
    ctx.set_tune(sid, **default)
    tune, _ = ctx.autotune(sid, spp=2, budget_ms=4000)
    assert tune["leaf_batch"] in (32, 8) and tune["shadow_leaf_batch"] in (32, 8)
    ctx.set_tune(sid, **default)
