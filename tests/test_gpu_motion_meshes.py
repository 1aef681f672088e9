"""Rays that meet several motion-blurred meshes in turn, and static triangles
between them: a lane keeps the object ray of the last motion mesh it met.
Against the CPU restatement in float."""
import dataclasses

import numpy as np
import pytest

from anacapa_b200 import api
from anacapa_b200 import scenes as S
from tests.test_gpu_queue_edges import check, random_rays

pytestmark = pytest.mark.gpu


def crowded(w, h, spp):
    """The motion scene with its moving meshes drawn together until their boxes
    overlap one another and a static sphere."""
    sc = S.motion(w, h, spp, 5)
    keys = []
    for k in sc.mesh_motion:
        if k:
            k = [(t, np.array(M, np.float32)) for t, M in k]
            for _, M in k:
                M[:3, 3] *= np.float32(0.35)
                M[1, 3] += np.float32(0.4)
        keys.append(k)
    return dataclasses.replace(sc, mesh_motion=keys)


@pytest.mark.parametrize("traversal", [api.ANA_TRAVERSAL_PER_RAY, api.ANA_TRAVERSAL_PERSISTENT],
                         ids=["per_ray", "persistent"])
def test_hits_of_overlapping_motion_meshes(gpu, restate_built, traversal):
    sc = crowded(64, 48, 1)
    rays = random_rays(60_001, 1.5, 41)
    rays[:, 1] += 0.5
    r = api.Renderer(traversal=traversal)
    try:
        r.upload(sc)
        check(r, restate_built.PoScene(sc, 32), rays)
    finally:
        r.close()


def test_frame_of_overlapping_motion_meshes(gpu, restate_built):
    sc = crowded(80, 60, 4)
    r = api.Renderer()
    try:
        r.upload(sc)
        r.render_scene(sc)
        f = r.film(sc.width, sc.height)
        ref, _ = restate_built.PoScene(sc, 32).render()
        rel = np.abs(f[..., :3] - ref[..., :3]) / np.maximum(np.abs(ref[..., :3]), 1e-3)
        assert (rel.max(-1) < 1e-3).mean() >= 0.95, float((rel.max(-1) < 1e-3).mean())
    finally:
        r.close()
