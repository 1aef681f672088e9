"""Ray queues whose length lies around the points where the persistent
schedule changes how it deals out entries (one per warp, a warp's 32 lanes,
ragged lengths), against the CPU restatement in float: the same ids and
distances, ties within 1e-6 relative t aside."""
import numpy as np
import pytest

from anacapa_b200 import api
from anacapa_b200 import scenes as S

pytestmark = pytest.mark.gpu

# Warps of the resident grids on 148 SMs: 5 blocks of 8 warps per SM (3 with curves)
WARPS = {"spheres": 148 * 5 * 8, "hair": 148 * 3 * 8}
SCENES = {"spheres": (lambda: S.throughput(64, 36, 1, 4, n_spheres=48, subdiv=2), 11.0),
          "hair": (lambda: S.hair(64, 36, 1, n_strands=3000), 1.6)}


def random_rays(n, extent, seed):
    rng = np.random.default_rng(seed)
    r = np.zeros((n, 8), np.float32)
    r[:, :3] = rng.uniform(-extent, extent, (n, 3))
    d = rng.normal(size=(n, 3))
    r[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    r[:, 3], r[:, 7] = 1e-4, 1e10
    return r


def check(r, po, rays):
    ids, t = po.trace(rays)
    g = r.trace(rays)
    gid = np.stack([g["hit"], g["mesh_id"], g["prim_id"], g["strand_id"]], 1)
    same = (gid == ids).all(1)
    tie = (ids[:, 0] == 1) & (g["hit"] == 1) & (np.abs(g["t"] - t) <= 1e-6 * np.abs(t))
    assert (same | tie).all()
    hit = same & (ids[:, 0] == 1)
    assert np.array_equal(g["t"][hit], t[hit].astype(np.float32))
    assert np.array_equal(r.trace(rays, occlusion=True)["hit"], ids[:, 0])


@pytest.mark.parametrize("scene", list(SCENES))
def test_queue_lengths(gpu, restate_built, scene):
    make, extent = SCENES[scene]
    sc, w = make(), WARPS[scene]
    po = restate_built.PoScene(sc, 32)
    rays = random_rays(32 * w + 33, extent, 21)
    r = api.Renderer()
    try:
        r.upload(sc)
        for n in (1, 31, 32, 33, w - 1, w, w + 1, 12 * w + 5, 32 * w, 32 * w + 33):
            check(r, po, rays[:n])
    finally:
        r.close()


@pytest.mark.parametrize("traversal", [api.ANA_TRAVERSAL_PER_RAY, api.ANA_TRAVERSAL_PERSISTENT],
                         ids=["per_ray", "persistent"])
def test_curve_rays_with_flat_components(gpu, restate_built, traversal):
    """Rays through strands with one or two direction components of 0, -0 or
    below 1e-9, which the curve boxes do not divide by, mixed with ordinary
    rays of either sign in one warp."""
    sc, _ = SCENES["hair"]
    sc = sc()
    rays = random_rays(4096, 1.6, 22)
    rng = np.random.default_rng(23)
    small = np.array([0.0, -0.0, 9e-10, -9e-10, 1e-9, -1e-9, 1e-12], np.float32)
    for k in range(3):
        rows = rng.random(len(rays)) < 0.35
        rays[rows, 4 + k] = rng.choice(small, rows.sum())
    keep = np.abs(rays[:, 4:7]).max(1) > 1e-3
    rays = rays[keep]
    rays[:, 4:7] /= np.linalg.norm(rays[:, 4:7].astype(np.float64), axis=1, keepdims=True)
    # aim half of them at strand control points
    cps = np.asarray(sc.control_points, np.float32).reshape(-1, 3)
    half = len(rays) // 2
    rays[:half, :3] = cps[rng.integers(0, len(cps), half)] - 0.5 * rays[:half, 4:7]
    po = restate_built.PoScene(sc, 32)
    r = api.Renderer(traversal=traversal)
    try:
        r.upload(sc)
        check(r, po, rays)
    finally:
        r.close()
