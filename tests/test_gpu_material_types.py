"""Uploaded scenes whose materials carry a type code beyond the known ones: such a surface has no
BSDF, so its paths pass through it, and they are shaded by the class of the index material
(which also covers the scenes where that class is otherwise empty)."""
import ctypes

import numpy as np
import pytest

import gianduia_b200 as G
from gianduia_b200 import scenes

pytestmark = [pytest.mark.gpu, pytest.mark.timeout(120)]

MATERIAL_BYTES = 160


@pytest.fixture(scope="module")
def ctx():
    c = G.GpuContext(0)
    yield c
    c.close()


@pytest.mark.parametrize("code", [5, 7, 0x80000000])
@pytest.mark.parametrize("batched", [True, False])
def test_unknown_material_type_passes_through(ctx, tmp_path, code, batched):
    hs = G.HostScene.load_xml(scenes.cornell(str(tmp_path), width=24, height=20, spp=3))
    types = [ctypes.c_uint32.from_address(hs.desc.materials + MATERIAL_BYTES * k) for k in range(hs.desc.num_materials)]
    assert len(types) > 2 and all(t.value < 4 for t in types)
    types[1].value = code   # host copy only
    sid = ctx.upload(hs)
    # one kernel for the whole list, without shade classes
    ctx.set_tune(sid, material_sort=0)
    ref, _, st0 = ctx.render_fixed(sid, spp=3, batched=batched)
    ctx.set_tune(sid, material_sort=1)
    got, _, st1 = ctx.render_fixed(sid, spp=3, batched=batched)
    assert st0["paths"] == st1["paths"] == 24 * 20 * 3
    assert np.array_equal(got, ref) and int(ref[..., :3].max()) > 0
    ctx.free_scene(sid)
