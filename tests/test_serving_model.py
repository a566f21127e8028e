"""The model of plain render times holds when the first passes of a render are not representative."""
import numpy as np
import pytest

from gianduia_b200 import serving


def test_plain_model_with_overlapping_passes(monkeypatch):
    def time_of(scene, res, spp, depth):
        # the first pass shows a whole path's length, each further one only its share
        return 1e-3 * (1.0 + 0.1 * depth) + 1e-8 * res * res * spp - (2e-4 if spp == 1 else 0.0)
    monkeypatch.setattr(serving, "_plain_time", lambda ctx, sid, integ, res, spp, depth: time_of(sid, res, spp, depth))
    reqs = serving.make_requests(200, seed=2)
    ids = {s: s for s in serving.SCENES}
    svc, info = serving.plain_service_model(None, ids, {s: 0 for s in serving.SCENES}, reqs, check=20)
    want = [time_of(r["scene"], r["res"], r["spp"], r["max_depth"]) for r in reqs]
    np.testing.assert_allclose(svc, want, rtol=1e-9)
    assert info["checked"] == 20 and info["max_rel_err"] == pytest.approx(0.0, abs=1e-9)
