"""Calls with host buffers give what the device-buffer calls give, at the sizes where the staged
copies change their way (one plain copy up to 256 KB, 1 MB chunks, a 32 MB stage), with pinned
buffers, and from several threads and contexts at once; non-finite refit positions are refused
and change nothing."""
import threading

import numpy as np
import pytest

import gianduia_b200 as G
from gianduia_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = G.GpuContext(0)
    yield c
    c.close()


def _device_hits(ctx, sid, rays):
    torch = pytest.importorskip("torch")
    r = torch.from_numpy(rays).cuda()
    out = torch.empty((rays.shape[0], 5), dtype=torch.float32, device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    ctx.trace_closest_dev(sid, r.data_ptr(), rays.shape[0], out.data_ptr(), s.cuda_stream)
    torch.cuda.synchronize()
    return out.cpu().numpy().view(G.HIT_DTYPE).reshape(-1)


@pytest.mark.parametrize("n", [1, 8192, 8193, 13108, 32768, 65537, 1048576, 1048577, 1700001])
def test_ray_batches(ctx, n):
    sid = ctx.upload(G.HostScene.from_triangles(scenes.random_triangles(2000, seed=3)))
    rays = scenes.random_rays(n, seed=n)
    ref = _device_hits(ctx, sid, rays)
    for _ in range(2):
        got = ctx.trace_closest(sid, rays)
        assert got.tobytes() == ref.tobytes()
    assert np.array_equal(ctx.trace_any(sid, rays), ref["inst"] >= 0)
    ctx.free_scene(sid)


def test_pinned_buffers(ctx):
    torch = pytest.importorskip("torch")
    sid = ctx.upload(G.HostScene.from_triangles(scenes.random_triangles(2000, seed=3)))
    pinned = torch.empty((100000, 8), dtype=torch.float32, pin_memory=True).numpy()
    pinned[:] = scenes.random_rays(100000, seed=4)
    assert ctx.trace_closest(sid, pinned).tobytes() == _device_hits(ctx, sid, pinned.copy()).tobytes()
    ctx.free_scene(sid)


def test_threads_and_contexts(ctx):
    other = G.GpuContext(0)
    jobs = []
    for k, c in enumerate((ctx, ctx, other, other)):
        tri = scenes.random_triangles(500 + k, seed=k)
        sid = c.upload(G.HostScene.from_triangles(tri))
        rays = scenes.random_rays(60000 + 7 * k, seed=20 + k)
        jobs.append((c, sid, rays, c.trace_closest(sid, rays)))
    bad = []

    def work(c, sid, rays, ref):
        for _ in range(20):
            if c.trace_closest(sid, rays).tobytes() != ref.tobytes():
                bad.append(sid)
    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not bad
    for c, sid, _, _ in jobs:
        c.free_scene(sid)
    other.close()


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_refit_refuses_non_finite_positions(ctx, value):
    tri = scenes.random_triangles(3001, seed=6).reshape(-1, 9)
    sid = ctx.upload(G.HostScene.from_triangles(tri))
    rays = scenes.random_rays(20000, seed=7)
    before = ctx.trace_closest(sid, rays)
    for at in (0, 3001 * 9 - 1, 13007):
        bad = tri.copy()
        bad.reshape(-1)[at] = value
        with pytest.raises(G.GndError) as e:
            ctx.refit_mesh(sid, 0, bad)
        assert e.value.status == G.GND_ERR_INVALID
    assert ctx.trace_closest(sid, rays).tobytes() == before.tobytes()
    ctx.free_scene(sid)
