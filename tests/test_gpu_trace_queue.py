"""The warp traversal of a ray queue (trace_rays) at the sizes where its
scheduling can go wrong: fewer rays than a warp, one more or less than the
leaf list's 32 and 64 entries, a share of the queue per warp below 32 lanes,
and queues larger than the grid; every primitive kind, deep stacks, rays that
share a leaf list with rays of very different length."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle as O
from pathtracer_gb300 import native as N
from pathtracer_gb300 import scene as S

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 63, 64, 65, 127, 4097, 34049, 200_003]


def _scene():
    """Mesh, rectangles, spheres, a box and curves."""
    sc, _ = S.hair_curves(40, seed=2)
    mat = sc.add_material(N.LAMBERTIAN, [0.5, 0.5, 0.5])
    sc.add_mesh(S.sphere_mesh(5, (0.3, 0.5, 0.2), 0.4, mat, displace=0.1, seed=1))
    sc.add_box((-1.5, 0.1, -1.2), (-0.9, 0.8, -0.6), mat)
    sc.add_sphere((-0.6, 0.6, 0.7), 0.35, mat)
    return sc


@pytest.fixture(scope="module")
def held(renderer):
    sc = _scene()
    sid = renderer.upload(sc)
    yield sid, O.OracleScene(sc)
    renderer.release(sid)


def _rays(n):
    rng = np.random.default_rng(n)
    o = rng.uniform(-2.5, 2.5, size=(n, 3))
    d = rng.uniform(-0.8, 0.9, size=(n, 3)) - o
    d[::7] = rng.normal(size=d[::7].shape)  # some that mostly miss
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([o, d], 1).astype(np.float32)


@pytest.mark.parametrize("n", SIZES)
def test_queue_sizes_match_oracle(renderer, held, n):
    sid, ref = held
    rays = _rays(n)
    t, prim, _ = renderer.trace_closest(sid, rays)
    t2, prim2 = ref.trace_closest(rays)
    # the tests restate one arithmetic, so hits agree but for exact ties
    assert ((prim >= 0) == (prim2 >= 0)).all()
    hit = prim2 >= 0
    assert np.all(np.abs(t[hit] - t2[hit]) <= 1e-5 * np.abs(t2[hit]))
    assert (prim == prim2).mean() >= (0.999 if n > 1000 else 1.0 - 1.0 / n)
    # any hit: occluded exactly where the closest hit lies in the interval
    tmax = np.where(np.arange(n) % 3 == 0, 0.5, 1e5).astype(np.float32)
    occ = renderer.trace_any(sid, rays, tmax, tmin=1e-4)
    assert np.array_equal(occ.astype(bool), hit & (t2 <= tmax))


def test_rays_of_one_leaf(renderer, held):
    """Every lane reaches the same leaf at the same turn: one ray, repeated."""
    sid, ref = held
    rays = np.repeat(_rays(64)[3:4], 1000, axis=0)
    t, prim, uv = renderer.trace_closest(sid, rays)
    assert (t == t[0]).all() and (prim == prim[0]).all() and (uv == uv[0]).all()
    assert prim[0] == ref.trace_closest(rays[:1])[1][0]
