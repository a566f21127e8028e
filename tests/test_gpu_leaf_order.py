"""Leaves whose box begins beyond a hit found before them are tested all the same: a triangle seen
almost edge-on reports distances far from its box (its determinant is close to zero), so it can
win against a hit in front of the box. Every mesh is one tree node whose leaves all pass the box
test before any triangle is tested; the nearest of all reported distances wins, as in the oracle."""
import numpy as np
import pytest

import gianduia_b200 as G
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

F = np.float32


def _tri_t(v, o, d):
    """Moller-Trumbore in float32, one ray per triangle; inf on a miss."""
    e1, e2, t = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0], o - v[:, 0]
    px, py, pz = (d[:, 1] * e2[:, 2] - d[:, 2] * e2[:, 1], d[:, 2] * e2[:, 0] - d[:, 0] * e2[:, 2],
                  d[:, 0] * e2[:, 1] - d[:, 1] * e2[:, 0])
    det = (e1[:, 0] * px + e1[:, 1] * py) + e1[:, 2] * pz
    inv = F(1) / det
    u = ((t[:, 0] * px + t[:, 1] * py) + t[:, 2] * pz) * inv
    qx, qy, qz = (t[:, 1] * e1[:, 2] - t[:, 2] * e1[:, 1], t[:, 2] * e1[:, 0] - t[:, 0] * e1[:, 2],
                  t[:, 0] * e1[:, 1] - t[:, 1] * e1[:, 0])
    w = ((d[:, 0] * qx + d[:, 1] * qy) + d[:, 2] * qz) * inv
    r = ((e2[:, 0] * qx + e2[:, 1] * qy) + e2[:, 2] * qz) * inv
    return np.where((np.abs(det) > 1e-8) & (u >= 0) & (u <= 1) & (w >= 0) & (u + w <= 1) & (r > 1e-4), r, np.inf)


def _entry(v, o, d):
    inv = F(1) / d
    a, b = (v.min(1) - o) * inv, (v.max(1) - o) * inv
    near, far = np.minimum(a, b).max(1), np.maximum(a, b).min(1)
    return np.where(near <= far, near, np.inf)


def _unit(x):
    return x / np.linalg.norm(x, axis=1, keepdims=True)


def _grazing(count, seed):
    """Triangles and rays where the box is entered later than the reported hit by more than 2e-4."""
    rng = np.random.default_rng(seed)
    n = 200000
    d = _unit(rng.normal(size=(n, 3)))
    s = _unit(np.cross(d, rng.normal(size=(n, 3))))
    up = np.cross(d, s)
    c = rng.uniform(1, 2, (n, 3))
    r = lambda lo, hi: rng.uniform(lo, hi, (n, 1))
    v = np.stack([c, c + d * r(.2, 1) + s * r(0, 1) + up * 1e-4 * r(-1, 1), c + d * r(.2, 1) - s * r(0, 1) + up * 1e-4 * r(-1, 1)],
                 1).astype(F)
    p = (v * rng.dirichlet((8, .3, .3), n)[:, :, None]).sum(1)
    o, d = (p - d * r(.5, 3)).astype(F), d.astype(F)
    with np.errstate(all="ignore"):
        t, e = _tri_t(v, o, d), _entry(v, o, d)
        gap = (e - t) / t
    pick = np.nonzero(np.isfinite(t) & np.isfinite(e) & (gap > 2e-4) & (gap < 1.0))[0][:count]
    assert len(pick) == count
    return v[pick], o[pick], d[pick], t[pick], gap[pick]


def test_grazing_triangle_behind_a_hit():
    count = 160
    v, o, d, t, gap = _grazing(count, 3)
    rng = np.random.default_rng(4)
    ctx = G.GpuContext(0)
    used = won = 0
    for k in range(count):
        w = d[k].astype(np.float64)
        s = _unit(np.cross(w, rng.normal(size=(1, 3))))[0]
        up = np.cross(w, s)

        def facing(at, size):
            c = o[k] + w * at
            return [c - s * size - up * size, c + s * size - up * size, c + up * size]
        mid = t[k] * (1.0 + 0.4 * gap[k])
        tri = [v[k]] + [facing(mid * (1.0 + 1e-6 * i), 1e-3 * gap[k]) for i in range(3)]
        for far in (40.0, -40.0):   # two leaves that the ray does not meet
            tri += [np.array(facing(far, 0.3)) + s * 9 + up * 0.1 * i for i in range(2)]
        tri = np.array(tri, F)
        hs = G.HostScene.from_triangles(tri)
        if hs.desc.num_nodes != 2:   # the top level and the mesh, a node each
            continue
        used += 1
        ray = np.concatenate([o[k], [1e-4], d[k], [np.inf]]).astype(F)[None]
        sid = ctx.upload(hs)
        got, ref = ctx.trace_closest(sid, ray), O.Scene.from_triangles(tri).trace(ray)
        assert got["prim"][0] == ref["prim"][0] and got["t"][0] == ref["t"][0], k
        won += int(ref["prim"][0] == 0)
        ctx.free_scene(sid)
    ctx.close()
    assert used >= 30 and won > used // 2
