"""Shading of short queues, where 2 or 4 lanes share a vertex's light samples:
a small window of a frame (few vertices per bounce) has the frame's bits, for
every count of light samples the split can meet (1, 2, 3, 4, 16: fewer than,
equal to and more than the lanes) and every kind of scene."""
from __future__ import annotations

import numpy as np
import pytest

from pathtracer_gb300 import native as N
from pathtracer_gb300 import scene as S

pytestmark = pytest.mark.gpu

SCENES = {
    "cornell": lambda: S.cornell_icosphere(3),
    "divergence": lambda: S.material_divergence(2, seed=3, aspect=1.0),
    "textured": lambda: S.textured_cornell(2),
    "glass": lambda: S.rough_glass(4, 64, 32),
}


@pytest.mark.parametrize("light_samples", [(1, 1), (2, 1), (3, 1), (2, 2), (4, 4)])
@pytest.mark.parametrize("name", sorted(SCENES))
def test_window_equals_frame(renderer, name, light_samples):
    sc, cam = SCENES[name]()
    sid = renderer.upload(sc)
    mis = name in ("cornell", "divergence")
    # 147 k paths: the first bounces fill the grid (no split), later ones and
    # the window's 1 k paths do not
    job = N.job_desc(sid, cam, 96, 96, 4, 4, 5, estimator=N.EST_NEE_MIS if mis else N.EST_REF_NEE, seed=7,
                     light_samples=light_samples)
    frame = renderer.render(job)
    job.width = job.height = 8
    job.crop_x, job.crop_y, job.full_width, job.full_height = 41, 37, 96, 96
    window = renderer.render(job)
    assert np.array_equal(window.view(np.uint32), np.ascontiguousarray(frame[37:45, 41:49]).view(np.uint32))
    renderer.release(sid)
