"""Traversal stacks beyond their 16 entries in shared memory: rays along a pile of
20 000 triangles whose boxes they all cross leave three entries per level of the
tree (10 levels and more).  Closest hits are the oracle's, occlusion is the closest
hit's verdict, in the world and in a moving object's frame."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle as O
from pathtracer_gb300 import native as N
from pathtracer_gb300 import scene as S

pytestmark = pytest.mark.gpu


def _pile(n, velocity):
    rng = np.random.default_rng(2)
    sc = S.Scene()
    mat = sc.add_material(N.LAMBERTIAN, [0.5, 0.5, 0.5])
    p = np.zeros((n, 3, 3))
    p[:, :, 2] = np.linspace(-4, 4, n)[:, None]
    p[:, :, :2] = [(-3, -3), (3, -3), (0, 3)]
    p += rng.uniform(-0.2, 0.2, p.shape)
    sc.add_mesh(S.Mesh(p.reshape(-1, 3).astype(np.float32), np.arange(3 * n, dtype=np.int32).reshape(n, 3), None, mat),
                velocity=velocity)
    sc.shutter_max = 1.0 if any(velocity) else 0.0
    return sc


@pytest.mark.parametrize("velocity", [(0.0, 0.0, 0.0), (0.0, 0.3, 0.0)], ids=["still", "moving"])
def test_deep_stacks_match_oracle(renderer, velocity):
    assert N.bvh_build(_pile(20000, (0.0, 0.0, 0.0)))["depth"] >= 10
    rng = np.random.default_rng(5)
    n = 3001
    d = np.concatenate([rng.uniform(-0.02, 0.02, (n, 2)), np.where(rng.random((n, 1)) < 0.5, 1.0, -1.0)], 1)
    # the triangles' boxes hold the corners that the triangles leave free
    o = np.concatenate([rng.uniform(-3.2, 3.2, (n, 2)), -5.0 * d[:, 2:]], 1)
    rays = np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)
    sid = renderer.upload(_pile(20000, velocity))
    t, prim, _ = renderer.trace_closest(sid, rays)
    t2, prim2 = O.OracleScene(_pile(20000, (0.0, 0.0, 0.0))).trace_closest(rays)
    hit = prim2 >= 0
    assert 0.2 < hit.mean() < 0.9
    assert np.array_equal(prim >= 0, hit) and (prim == prim2).mean() > 0.999
    assert np.all(np.abs(t[hit] - t2[hit]) <= 1e-5 * np.abs(t2[hit]))
    occ = renderer.trace_any(sid, rays, np.full(n, 1e5, np.float32), 1e-4)
    assert np.array_equal(occ.astype(bool), hit)
    renderer.release(sid)
