"""Occlusion through the any-hit rays' own top of the BVH: it must equal the
closest hit's verdict (another tree top) on scenes whose tops differ most from
the built tree -- many objects in insertion order, moving objects, one mesh
only, one node only."""
from __future__ import annotations

import numpy as np
import pytest

from pathtracer_gb300 import native as N
from pathtracer_gb300 import scene as S

pytestmark = pytest.mark.gpu


def _spheres(n):
    rng = np.random.default_rng(4)
    sc = S.Scene()
    mat = sc.add_material(N.LAMBERTIAN, [0.5, 0.5, 0.5])
    for _ in range(n):
        sc.add_sphere(tuple(rng.uniform(-3, 3, size=3)), float(rng.uniform(0.05, 0.3)), mat)
    return sc


SCENES = {
    "one_sphere": lambda: _spheres(1),
    "five_spheres": lambda: _spheres(5),
    "700_spheres": lambda: _spheres(700),
    "one_mesh": lambda: S.rough_glass(5, 8, 4)[0],
    "curves": lambda: S.hair_curves(60)[0],
    "objects": lambda: S.material_divergence(2, seed=1)[0],
    "moving": lambda: S.with_motion(S.material_divergence(2, seed=1)[0], 3),
}


@pytest.mark.parametrize("name", sorted(SCENES))
def test_occlusion_equals_closest_hit(renderer, name):
    sid = renderer.upload(SCENES[name]())
    rng = np.random.default_rng(9)
    n = 20011
    o = rng.uniform(-4, 4, size=(n, 3))
    d = rng.uniform(-3, 3, size=(n, 3)) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.concatenate([o, d], 1).astype(np.float32)
    t, prim, _ = renderer.trace_closest(sid, rays, 1e-3, 1e5)
    for far in (1.5, 1e5):
        occ = renderer.trace_any(sid, rays, np.full(n, far, np.float32), 1e-3)
        assert np.array_equal(occ.astype(bool), (prim >= 0) & (t <= np.float32(far)))
    renderer.release(sid)
