"""The Disney vertices' front-face and inside hits are sorted into bins of
their own, from the geometric side of the hit: a window of a frame, whose
vertices are sorted among others, has the frame's bits, and the frame agrees
with the oracle, for every kind of primitive the side is taken from (mesh,
sphere, rectangle, flipped faces, moving objects), with the neighbouring
families (Phong, hair) in the scene."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle as O
from pathtracer_gb300 import native as N
from pathtracer_gb300 import scene as S

pytestmark = pytest.mark.gpu

DISNEY = [0.8, 0.4, 0.2, 0.3, 0.4, 0.3, 0.5, 0.4, 0.2, 0.1, 0.4, 0.5, 0.5, 0.7, 1.5]


def scene_of(kind):
    sc = S.Scene()
    dis = sc.add_material(N.DISNEY, DISNEY)
    hair = sc.add_material(N.HAIR, [0, 0, 0, 0.0, 1.55, 0.3, 0.3, 0.035, 1.0, 0.0], N.FLAG_MELANIN)
    phong = sc.add_material(N.PHONG, [0.5, 0.4, 0.3, 0.2, 0.2, 0.2, 0, 0, 0, 20.0])
    light = sc.add_material(N.DIFFUSE_EMITTER, [1.0, 0.9, 0.8, 12.0])
    sc.add_quad(1, -1.0, -4.0, 4.0, -4.0, 4.0, phong)
    sc.add_sphere((2.0, 3.0, -2.0), 0.6, light)
    sc.add_sphere((-1.4, -0.4, 0.6), 0.5, hair)
    if kind in ("mesh", "moving"):
        v, f = S.icosphere(3)
        sc.add_mesh(S.Mesh(v.astype(np.float32), f.astype(np.int32), v.astype(np.float32), dis))
    elif kind == "rectangle":
        for k in range(3):
            sc.add_quad(k, 0.3 * k - 0.2, -1.0, 1.0, -0.8, 1.2, dis, flip=k & 1)
    else:
        sc.add_sphere((0.0, 0.0, 0.0), 1.0, dis, flip=int(kind == "flipped"))
    if kind == "moving":
        sc = S.with_motion(sc, 4)
    shutter = 0.5 if kind == "moving" else 0.0
    return sc, S.camera((0.4, 1.2, -4.0), (-0.1, -0.3, 1.0), 45.0, 1.0, shutter=shutter)


@pytest.mark.parametrize("kind", ["mesh", "sphere", "flipped", "rectangle", "moving"])
def test_sides_of_disney_hits(renderer, kind):
    sc, cam = scene_of(kind)
    sid = renderer.upload(sc)
    job = N.job_desc(sid, cam, 48, 48, 4, 4, 6, estimator=N.EST_NEE_MIS, seed=3)
    frame = renderer.render(job)
    assert np.isfinite(frame).all()
    job.width = job.height = 8
    job.crop_x, job.crop_y, job.full_width, job.full_height = 19, 21, 48, 48
    window = renderer.render(job)
    assert np.array_equal(window.view(np.uint32), np.ascontiguousarray(frame[21:29, 19:27]).view(np.uint32))
    job.width = job.height = 48
    job.crop_x = job.crop_y = job.full_width = job.full_height = 0
    job.scene = 0
    ref, _ = O.render(sc, job)
    close = np.isclose(frame, ref, rtol=1e-3, atol=1e-4).all(-1)
    assert close.mean() > 0.95, close.mean()
    renderer.release(sid)
