"""Ray queues whose length lies around the points where the persistent
schedule changes how it deals out entries (one per warp, a warp's 32 lanes,
ragged lengths), against the CPU restatement in float: the same ids and
distances, ties within 1e-6 relative t aside."""
import dataclasses
import hashlib

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


@pytest.mark.parametrize("traversal", [api.ANA_TRAVERSAL_PER_RAY, api.ANA_TRAVERSAL_PERSISTENT],
                         ids=["per_ray", "persistent"])
@pytest.mark.parametrize("scale,shift,stretch", [(1.0, 0.0, 1.0), (1.0, 1000.0, 1.0), (1e-3, 0.0, 1.0),
                                                 (500.0, 0.0, 1.0), (1.0, 0.0, 0.37), (1.0, 0.0, 25.0)],
                         ids=["plain", "far_from_origin", "tiny", "large", "short_direction", "long_direction"])
def test_rays_at_ribbon_edges(gpu, restate_built, scale, shift, stretch, traversal):
    """Rays past strands at distances around the half-width, where a segment
    may only be rejected unseen if no leaf of its walk is hit: strands far from
    the origin, tiny and large, thin and wide, against the restatement. For
    directions that are not of unit length a ribbon's distance and a box's are
    in different units, and what is found depends on the order of the visits;
    there the answers are those of the walk without any rejection, recorded."""
    sc = S.hair(64, 36, 1, n_strands=600)
    cps = np.asarray(sc.control_points, np.float32).reshape(-1, 3) * np.float32(scale) + np.float32(shift)
    widths = np.asarray(sc.widths, np.float32) * np.float32(scale)
    widths[::4] *= np.float32(20.0)
    sc = dataclasses.replace(sc, control_points=cps, widths=widths, area_lights=[])
    rng = np.random.default_rng(24)
    n = 1 << 15
    at = rng.integers(0, 600, n) * 13 + rng.integers(1, 12, n)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    p = cps.astype(np.float64)
    side = np.cross(d, p[at + 1] - p[at - 1])
    side /= np.maximum(np.linalg.norm(side, axis=1, keepdims=True), 1e-30)
    off = 0.5 * widths.reshape(-1, 2)[at // 13].mean(1) * rng.choice([0.0, 0.3, 0.9, 0.999, 1.0, 1.001, 1.1, 1.5], n)
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = p[at] + side * off[:, None] - d * (scale * rng.uniform(0.01, 2.0, (n, 1)))
    rays[:, 4:7] = d * stretch
    rays[:, 3], rays[:, 7] = 1e-4 * scale, 1e10
    r = api.Renderer(traversal=traversal)
    try:
        r.upload(sc)
        if stretch == 1.0:
            check(r, restate_built.PoScene(sc, 32), rays)
        else:
            found = [hashlib.sha1(r.trace(rays, occlusion=o).tobytes()).hexdigest()[:10] for o in (False, True)]
            assert found == {0.37: ["47406624bd", "de8dd33e3e"], 25.0: ["ac511829ec", "f4250bde8c"]}[stretch]
    finally:
        r.close()
