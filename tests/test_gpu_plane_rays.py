"""Hits without an order: a ray in the plane of a rectangle, or along the axis of
a straight curve, divides 0 by 0 there, and the reference's leaf loop takes that
t = NaN as a hit where the ray meets the bounds, and after it any other.  One
rectangle, one box (six faces of one leaf) and one curve have one order of tests
only, so every answer is the oracle's, bit for bit: alone and among other rays,
in the world and in a moving object's frame, with and without far curves in the
scene (whose nodes' coarse grids let rays through to the near leaf).  Where the order comes from the tree, a ray's answer does not depend
on the rays it is traced with."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle as O
from pathtracer_gb300 import native as N
from pathtracer_gb300 import scene as S

pytestmark = pytest.mark.gpu


def _scene(name, kind):
    sc = S.Scene()
    mat = sc.add_material(N.LAMBERTIAN, [0.5, 0.5, 0.5])
    vel = (0.0, 0.0, 0.0)
    if kind == "moving":
        vel, sc.shutter_max = (0.25, 0.0, 0.0), 1.0
    if name == "rectangle":
        sc.add_quad(0, 1.0, -1, 1, -1, 1, mat, velocity=vel)
    elif name == "curve":
        sc.add_curve([(0, y, 0) for y in (-1, -0.5, 0.5, 1)], 0.3, 0.3, mat, velocity=vel)
    else:
        sc.add_box((-1, -1, -1), (1, 1, 1), mat, velocity=vel)
    if kind == "curves":  # out of every ray's reach
        sc.add_curve([(900, 900, 900 + k) for k in range(4)], 0.01, 0.01, mat)
    return sc


def _rays(n):
    """Origins on a grid that the planes are part of, axis-parallel parts."""
    rng = np.random.default_rng(n)
    o = rng.integers(-12, 13, (n, 3)) * 0.25
    d = rng.normal(size=(n, 3))
    d[np.arange(n), rng.integers(0, 3, n)] = 0
    one = rng.random(n) < 0.3
    d[one, rng.integers(0, 3, one.sum())] = 0
    d[np.abs(d).sum(1) == 0] = (0, 0, 1)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([o, d], 1).astype(np.float32)


def _clear(rays, lo, hi, margin=0.05):
    """Rays that meet or miss the box [lo, hi] by a margin, but for one axis
    that they do not move along: a rectangle or a box is tested, and its NaN
    accepted, only where its bounding box is met."""
    o, d = rays[:, :3].astype(np.float64), rays[:, 3:].astype(np.float64)
    lo, hi = np.asarray(lo, np.float64), np.asarray(hi, np.float64)
    edge = (d == 0) & ((o == lo) | (o == hi))

    def meets(m):
        near, far = np.full(len(o), 1e-4), np.full(len(o), 1e5)
        for a in range(3):
            with np.errstate(divide="ignore", invalid="ignore"):
                t = np.sort([(lo[a] - m - o[:, a]) / d[:, a], (hi[a] + m - o[:, a]) / d[:, a]], axis=0)
            still = (o[:, a] > lo[a] - m) & (o[:, a] < hi[a] + m) | edge[:, a]
            t = np.where(d[:, a] == 0, np.where(still, -np.inf, np.inf) * np.array([[1], [-1]]), t)
            near, far = np.maximum(near, t[0]), np.minimum(far, t[1])
        return near < far

    return (meets(margin) == meets(-margin)) & (edge.sum(1) < 2)


@pytest.mark.parametrize("kind", ["plain", "moving", "curves"])
@pytest.mark.parametrize("name", ["rectangle", "box", "curve"])
def test_rays_in_a_plane_match_oracle(renderer, name, kind):
    ref = O.OracleScene(_scene(name, "plain"))
    sid = renderer.upload(_scene(name, kind))
    rays = _rays(20011)
    if name == "curve":
        rays[:, 3:] = np.where(np.arange(len(rays))[:, None] % 2 == 0, 1, -1) * np.array([0, 1, 0], np.float32)
    lo, hi = {"rectangle": ((1, -1, -1), (1, 1, 1)), "box": ((-1, -1, -1), (1, 1, 1)),
              "curve": ((-0.3, -1.3, -0.3), (0.3, 1.3, 0.3))}[name]
    rays = rays[_clear(rays, lo, hi)]
    t2, prim2 = ref.trace_closest(rays)
    plane = np.flatnonzero((prim2 >= 0) & ~(t2 <= 1e5))
    assert plane.size > 20
    t, prim, uv = renderer.trace_closest(sid, rays)
    assert np.array_equal(prim, prim2) and np.array_equal(t, t2, equal_nan=True)
    occ = renderer.trace_any(sid, rays, np.full(len(rays), 1e5, np.float32), 1e-4)
    assert np.array_equal(occ.astype(bool), prim2 >= 0)
    hit = renderer.intersect(sid, rays)
    assert np.array_equal(hit[1], prim2) and np.array_equal(hit[0], t2, equal_nan=True)
    for m in (1, 2, 33):  # few rays, all of them in planes
        t, prim, _ = renderer.trace_closest(sid, rays[plane[:m]])
        assert np.array_equal(prim, prim2[plane[:m]]) and np.array_equal(t, t2[plane[:m]], equal_nan=True)
    renderer.release(sid)


def test_answers_do_not_depend_on_the_queue(renderer):
    rng = np.random.default_rng(3)
    sc = S.Scene()
    mat = sc.add_material(N.LAMBERTIAN, [0.5, 0.5, 0.5])
    for i in range(300):
        k, a = rng.integers(-12, 13) * 0.25, rng.integers(-12, 9, 2) * 0.25
        b = a + rng.integers(1, 12, 2) * 0.25
        sc.add_quad(i % 3, float(k), float(a[0]), float(b[0]), float(a[1]), float(b[1]), mat)
    for _ in range(60):
        lo = rng.integers(-12, 9, 3) * 0.25
        sc.add_box(tuple(lo), tuple(lo + rng.integers(1, 8, 3) * 0.25), mat)
    sid = renderer.upload(sc)
    rays = _rays(20011)
    t, prim, _ = renderer.trace_closest(sid, rays)
    assert np.isnan(t).sum() > 100
    for m in (1, 7, 64, 1000):
        t1, prim1, _ = renderer.trace_closest(sid, rays[:m])
        assert np.array_equal(prim1, prim[:m]) and np.array_equal(t1, t[:m], equal_nan=True)
    perm = rng.permutation(rays.shape[0])
    t1, prim1, _ = renderer.trace_closest(sid, rays[perm])
    assert np.array_equal(prim1, prim[perm]) and np.array_equal(t1, t[perm], equal_nan=True)
    renderer.release(sid)


@pytest.mark.parametrize("where", [0.0, 100.0])
def test_unnormalised_directions_do_not_depend_on_the_queue(renderer, where):
    """t is a distance on a rectangle or sphere and a multiple of the direction
    on a triangle (and in the boxes): a ray's hit still depends on the ray alone."""
    rng = np.random.default_rng(8)
    sc = S.Scene()
    mat = sc.add_material(N.LAMBERTIAN, [0.5, 0.5, 0.5])
    for i in range(300):
        k, a = where + rng.integers(-8, 9) * 0.25, where + rng.integers(-8, 7, 2) * 0.25
        b = a + rng.integers(1, 12, 2) * 0.25
        sc.add_quad(i % 3, float(k), float(a[0]), float(b[0]), float(a[1]), float(b[1]), mat)
    for _ in range(50):
        sc.add_sphere(tuple(where + rng.uniform(-2, 2, 3)), float(rng.uniform(0.1, 0.5)), mat)
    sc.add_mesh(S.sphere_mesh(3, (where,) * 3, 1.5, mat, displace=0.2, seed=1))
    sid = renderer.upload(sc)
    n = 20011
    o = where + rng.uniform(-4, 4, (n, 3))
    d = (where + rng.uniform(-2, 2, (n, 3)) - o) * np.exp(rng.uniform(-3, 3, (n, 1)))
    rays = np.concatenate([o, d], 1).astype(np.float32)
    t, prim, _ = renderer.trace_closest(sid, rays)
    assert (prim >= 0).mean() > 0.5
    perm = rng.permutation(n)
    for sel in (perm, perm[:3001], perm[:64], perm[:5]):
        t1, prim1, _ = renderer.trace_closest(sid, rays[sel])
        assert np.array_equal(prim1, prim[sel]) and np.array_equal(t1, t[sel])
    hit = renderer.intersect(sid, rays[perm])
    assert np.array_equal(hit[1], prim[perm]) and np.array_equal(hit[0], t[perm])
    renderer.release(sid)
