"""Served films of many sizes finishing together (more than there are stages to leave through), and
mixes of scenes that need more round graphs than the engine keeps."""
import ctypes

import numpy as np
import pytest

import gianduia_b200 as G
from gianduia_b200 import scenes

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(300)]


def test_films_of_many_sizes(tmp_path):
    ctx = G.GpuContext(0)
    sid = ctx.upload(G.HostScene.load_xml(scenes.cornell(str(tmp_path), width=64, height=64, spp=2)))
    rng = np.random.default_rng(5)
    jobs = [dict(width=int(w), height=int(h), spp=1, max_depth=3) for w, h in rng.integers(1, 500, (24, 2))]
    for _ in range(2):   # the second time into stages that exist
        ids = [ctx.submit(sid, **j) for j in jobs]
        films = [ctx.wait(i, timeout_ms=30000) for i in ids]
        for (film, st), j in zip(films, jobs):
            assert st["state"] == "done"
            assert np.array_equal(film[..., :4], ctx.render(sid, **j)[0][..., :4]), j
    ctx.close()


def test_more_graphs_than_are_kept(tmp_path):
    hs = G.HostScene.load_xml(scenes.cornell(str(tmp_path), width=16, height=12, spp=1))
    kinds = [ctypes.c_uint32.from_address(hs.desc.materials + 160 * k) for k in range(hs.desc.num_materials)]
    assert len(kinds) >= 4
    ctx, plain = G.GpuContext(0), G.GpuContext(0)
    ids = []
    for mask in range(1, 32):   # the material types (of which 4: no BSDF) that the scene holds
        types = [t for t in range(5) if mask & (1 << t)]
        for k, m in enumerate(kinds):
            m.value = types[k % len(types)]   # host copy only
        pair = ctx.upload(hs), plain.upload(hs)
        ctx.set_tune(pair[0], round_iters=4)   # as the server's: another setting drops the graphs
        plain.set_tune(pair[1], graphs=0)
        ids.append(pair)
    for integrator in (0, 1):   # 31 class sets x 2 integrators, rendered and served: 124 graphs
        for a, b in ids:
            job = dict(spp=1, max_depth=3, integrator=integrator)
            ref = plain.render(b, **job)[0]
            assert np.array_equal(ctx.render(a, **job)[0][..., :4], ref[..., :4])
            film, st = ctx.wait(ctx.submit(a, **job), timeout_ms=30000)
            assert st["state"] == "done" and np.array_equal(film[..., :4], ref[..., :4])
    ctx.close()
    plain.close()
