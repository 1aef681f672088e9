"""Device-built subtrees of one warp (at most 128 triangles) around the warp's
32 lanes and its 128 triangles: the host build's bytes, for scattered and
overlapping triangles, equal centroids (the median fallback) and coordinates of
both zeros, which the sequential minimum keeps in order."""
import numpy as np
import pytest

from anacapa_b200 import api
from anacapa_b200 import scenes as S

pytestmark = pytest.mark.gpu


def soup(n, kind, seed):
    rng = np.random.default_rng(seed)
    p = rng.uniform(-1.0, 1.0, (n, 1, 3)) + rng.uniform(-0.2, 0.2, (n, 3, 3))
    if kind == "grid":  # few distinct centroids
        p = np.round(p * 2.0) / 2.0 + np.array([[0.0, 0.0, 0.0], [0.25, 0.0, 0.1], [0.0, 0.25, 0.05]])
    if kind == "zeros":  # planes through the origin, zeros of both signs
        p = np.where(rng.random(p.shape) < 0.4, np.where(rng.random(p.shape) < 0.5, 0.0, -0.0), p)
    if kind == "equal":
        p[:] = p[:1]
    b = S._Builder()
    m = b.material(S.Material(S.MAT_LAMBERT, albedo=(0.5, 0.5, 0.5)))
    b.mesh(p.reshape(-1, 3), np.arange(3 * n).reshape(n, 3), m)
    return b.scene("soup", area_lights=[], env_radiance=(1.0, 1.0, 1.0), width=4, height=4, spp=1)


@pytest.mark.parametrize("leaf", [0, 1, 8], ids=["default", "leaf1", "leaf8"])
@pytest.mark.parametrize("kind", ["scattered", "grid", "zeros", "equal"])
def test_small_subtrees_match_the_host_build(gpu, kind, leaf):
    r = api.Renderer()
    try:
        for n in (1, 2, 4, 5, 8, 9, 31, 32, 33, 63, 64, 65, 96, 97, 127, 128):
            sc = soup(n, kind, n)
            r.upload(sc, device_build=True, max_leaf_tris=leaf)
            assert r.scene_digest() == api.Prepared(sc, max_leaf_tris=leaf).digest, n
    finally:
        r.close()
