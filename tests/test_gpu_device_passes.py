"""Plain renders without a progress callback: the device releases the passes, whole, as path
slots free up. The exact film equals the batched one whatever the number of passes, the
window and the order of release; a cancelled render holds whole passes only; and scenes of one
material class, which skip the classification, render the same film with it."""
import threading
import time

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


@pytest.mark.parametrize("spp,window", [(1, None), (2, None), (7, None), (3, (5, 9, 6, 10)), (64, (11, 3, 12, 4)), (9, (0, 17, 33, 64))])
def test_exact_film_of_device_released_passes(ctx, tmp_path, spp, window):
    sid = ctx.upload(G.HostScene.load_xml(scenes.cornell(str(tmp_path), width=65, height=64)))
    plain, _, st = ctx.render_fixed(sid, spp=spp, first_pass=3, window=window)
    batched, _, sb = ctx.render_fixed(sid, spp=spp, first_pass=3, window=window, batched=True)
    npix = 65 * 64 if window is None else (window[2] - window[0]) * (window[3] - window[1])
    assert st["paths"] == sb["paths"] == npix * spp and st["passes"] == spp
    assert np.array_equal(plain, batched)
    ctx.set_tune(sid, material_sort=0)
    assert np.array_equal(ctx.render_fixed(sid, spp=spp, first_pass=3, window=window)[0], plain)
    ctx.set_tune(sid, material_sort=1, graphs=0)
    assert np.array_equal(ctx.render_fixed(sid, spp=spp, first_pass=3, window=window)[0], plain)
    ctx.free_scene(sid)


def test_progress_callback_sees_every_pass(ctx, tmp_path):
    sid = ctx.upload(G.HostScene.load_xml(scenes.cornell(str(tmp_path), width=48, height=40)))
    seen = []
    film, st = ctx.render(sid, spp=5, callback=lambda s, f: seen.append((s, float(f[..., 3].sum()))))
    assert [s for s, _ in seen] == [0, 1, 2, 3, 4] and st["passes"] == 5
    assert all(abs(w - (s + 1) * 48 * 40) < 1.0 for s, w in seen)
    assert np.array_equal(ctx.render(sid, spp=5)[0][..., :4], film[..., :4])
    ctx.free_scene(sid)


def test_cancel_leaves_whole_passes(ctx, tmp_path):
    sid = ctx.upload(G.HostScene.load_xml(scenes.cornell(str(tmp_path), width=256, height=256)))
    film = np.zeros((256, 256, 7), np.float32)
    result = []

    def work():
        try:
            ctx.render(sid, spp=200000, film=film)
            result.append(None)
        except G.GndError as e:
            result.append(e.status)
    t = threading.Thread(target=work)
    t.start()
    time.sleep(0.3)
    ctx.cancel()
    t.join(60)
    assert result == [G.GND_ERR_CANCELLED]
    w = film[..., 3]
    passes = np.median(w)
    assert passes >= 1 and passes == np.round(passes) and passes < 200000
    # a sample on a whole coordinate also counts for its neighbour: a few pixels per million samples
    assert np.mean(w == passes) > 0.95 and np.all(w >= passes - 0.5)
    ctx.free_scene(sid)
