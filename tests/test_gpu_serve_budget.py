"""Jobs under an HBM budget: a job that submit accepts (it fits alone, with its scenes and the path
pool) runs, whatever films, film stages and pools earlier work left idle; films stay exact."""
import re

import numpy as np
import pytest

import gianduia_b200 as G
from gianduia_b200 import scenes

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(300)]

WAIT_MS = 20000


@pytest.fixture()
def setup(tmp_path):
    ctx = G.GpuContext(0)
    ctx.serve_tune(pool_log2=18)
    hs = G.HostScene.load_xml(scenes.cornell(str(tmp_path), width=64, height=64, spp=2))
    yield ctx, ctx.upload(hs), hs
    ctx.close()


def _alone(ctx, sid, **job):
    """Bytes the job needs alone, as the refusal states them."""
    ctx.set_hbm_budget(1)
    with pytest.raises(G.GndError) as e:
        ctx.submit(sid, **job)
    assert e.value.status == G.GND_ERR_BUDGET
    return int(re.search(r"job needs (\d+) bytes", str(e.value)).group(1))


def _check(ctx, sid, jid, **job):
    film, st = ctx.wait(jid, timeout_ms=WAIT_MS)
    assert st["state"] == "done"
    ref, _ = ctx.render(sid, **job)
    assert np.array_equal(film[..., :4], ref[..., :4])


def test_jobs_after_a_burst(setup):
    ctx, sid, _ = setup
    big = dict(width=400, height=300, spp=2, max_depth=4)
    ids = [ctx.submit(sid, **big) for _ in range(9)]   # more films at once than there are stages
    for j in ids:
        assert ctx.wait(j, timeout_ms=WAIT_MS)[1]["state"] == "done"
    # exactly what each job needs alone: the same size, a smaller one, one larger than any before
    for job in (big, dict(big, width=33, height=21), dict(big, width=501, height=333)):
        ctx.set_hbm_budget(_alone(ctx, sid, **job))
        _check(ctx, sid, ctx.submit(sid, **job), **job)


def test_queued_jobs_take_turns(setup):
    ctx, sid, _ = setup
    sizes = [(300, 200), (64, 48), (320, 240), (16, 16), (200, 301), (320, 240), (1, 1)]
    jobs = [dict(width=w, height=h, spp=2, max_depth=4) for w, h in sizes]
    ctx.set_hbm_budget(max(_alone(ctx, sid, **j) for j in jobs))
    ids = [ctx.submit(sid, **j) for j in jobs]
    for j, job in zip(ids, jobs):
        film, st = ctx.wait(j, timeout_ms=WAIT_MS)
        assert st["state"] == "done" and st["samples_done"] == job["width"] * job["height"] * 2
    ctx.set_hbm_budget(0)


def test_job_after_renders_with_larger_pools(setup):
    ctx, sid, hs = setup
    ctx.set_tune(sid, pool_log2=20)
    ctx.render(sid, width=512, height=512, spp=8, batched=True)   # a pool of 2^20 slots and its film
    job = dict(width=64, height=64, spp=2, max_depth=4)
    ctx.set_hbm_budget(_alone(ctx, sid, **job))
    _check(ctx, sid, ctx.submit(sid, **job), **job)
    # a pool smaller than the serving one grows by the difference
    other = G.GpuContext(0)
    sid2 = other.upload(hs)
    other.serve_tune(pool_log2=18)
    other.render(sid2, width=300, height=200, spp=2)
    other.set_hbm_budget(_alone(other, sid2, **job))
    _check(other, sid2, other.submit(sid2, **job), **job)
    other.close()
