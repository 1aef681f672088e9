"""Workloads that stand for what users of the renderer have it do.

Every case goes through the public binding (`anacapa_b200.api`,
`anacapa_b200.diff`) on scenes of the repository's generators, over the sizes
of its configurations, tests and benchmark:

  frame     one render pass and the read of its film (`Renderer.render`,
            `Renderer.film`, with AOVs `Renderer.aovs`)
  batch     several scenes rendered in one graph-replayed launch sequence
            (`Renderer.render_batch`) and the read of every film
  gradient  one optimisation step's forward and backward pass through the
            autograd function (`diff.render`)
  trace     a batch of ray queries on host buffers (`Renderer.trace`)
  pick      a small query that may not allocate (`Renderer.trace_noalloc`)
  open      a scene handed over and its first preview pass
            (`Renderer.upload(device_build=True)`, `Renderer.render`)

A case holds the scene ("scene", its primitive count "n") and the call's sizes.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from anacapa_b200 import api, diff
from anacapa_b200 import scenes as S

# Rays of one query whose exact answer is computed by testing every triangle
EXACT_TESTS = 4e9


def listed():
    return [
        # a pick or marquee query of an interactive viewer, beside whatever else runs
        {"name": "pick 64 rays", "kind": "pick", "scene": "spheres", "n": 938, "rays": 64, "occlusion": False},
        # the small closed box: tests, thumbnails, look development
        {"name": "cornell 256x256x16", "kind": "frame", "scene": "cornell", "n": 0, "width": 256, "height": 256,
         "spp": 16, "depth": 8, "aovs": False},
        # one progressive pass of an interactive viewer on an ordinary scene
        {"name": "preview 960x540x1", "kind": "frame", "scene": "spheres", "n": 938, "width": 960, "height": 540,
         "spp": 1, "depth": 12, "aovs": False},
        # the final frame at its production size: 5.2 M triangles under an HDR dome
        {"name": "spheres 1920x1080x64", "kind": "frame", "scene": "spheres", "n": 4096, "width": 1920,
         "height": 1080, "spp": 64, "depth": 12, "aovs": False},
        # curves: 200 k strands, one pass of a progressive final frame
        {"name": "hair 1280x720x8", "kind": "frame", "scene": "hair", "n": 200_000, "width": 1280, "height": 720,
         "spp": 8, "depth": 10, "aovs": False},
        # glass and alpha masks at an odd, cropped size
        {"name": "glass 1279x719x16", "kind": "frame", "scene": "glass", "n": 0, "width": 1279, "height": 719,
         "spp": 16, "depth": 8, "aovs": False},
        # motion blur with the denoiser's AOVs
        {"name": "motion aov 1280x720x16", "kind": "frame", "scene": "motion", "n": 0, "width": 1280, "height": 720,
         "spp": 16, "depth": 6, "aovs": True},
        # variants of one scene with uneven resolutions, spp and depths (dataset generation)
        {"name": "batch of 24 variants", "kind": "batch", "scene": "cornell", "n": 24},
        # inverse rendering: one step on the differentiable scene
        {"name": "gradient 512x512x16", "kind": "gradient", "scene": "differentiable", "n": 5, "width": 512,
         "height": 512, "spp": 16, "depth": 8},
        # closest hits of incoherent rays (baking, probes), host buffers in and out
        {"name": "trace 1M closest", "kind": "trace", "scene": "spheres", "n": 938, "rays": 1 << 20,
         "occlusion": False},
        # occlusion of incoherent segments against curves, a ragged count
        {"name": "trace 200k hair occlusion", "kind": "trace", "scene": "hair", "n": 200_000, "rays": 200_001,
         "occlusion": True},
        # opening a scene of 1.2 M triangles and seeing its first pass
        {"name": "open 938 spheres", "kind": "open", "scene": "spheres", "n": 938, "width": 480, "height": 270,
         "spp": 1, "depth": 12, "aovs": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _scene_and_size(rng, scenes):
    scene = rng.choice(scenes)
    n = {"spheres": lambda: _log_int(rng, 16, 4096), "hair": lambda: _log_int(rng, 2000, 200_000)}.get(
        scene, lambda: 0)()
    return scene, n


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "batch", "gradient", "trace", "trace", "pick", "open"])
    if kind == "frame":
        scene, n = _scene_and_size(rng, ["cornell", "spheres", "spheres", "hair", "glass", "motion", "sunlit"])
        width, height = _log_int(rng, 64, 1920), _log_int(rng, 48, 1080)
        most = {"hair": 7.0e6, "spheres": 6.0e7}.get(scene, 3.0e7)
        spp = _log_int(rng, 1, max(1.0, min(64.0, most / (width * height))))
        return {"kind": kind, "scene": scene, "n": n, "width": width, "height": height, "spp": spp,
                "depth": rng.randint(2, 12), "aovs": rng.random() < 0.3}
    if kind == "batch":
        return {"kind": kind, "scene": "cornell", "n": rng.randint(2, 24)}
    if kind == "gradient":
        width, height = _log_int(rng, 64, 512), _log_int(rng, 64, 512)
        return {"kind": kind, "scene": "differentiable", "n": rng.randint(2, 5), "width": width, "height": height,
                "spp": _log_int(rng, 1, 16), "depth": rng.randint(2, 8)}
    if kind == "open":
        return {"kind": kind, "scene": "spheres", "n": _log_int(rng, 16, 2000), "width": _log_int(rng, 160, 640),
                "height": _log_int(rng, 90, 360), "spp": rng.randint(1, 4), "depth": rng.randint(2, 12),
                "aovs": False}
    scene, n = _scene_and_size(rng, ["cornell", "spheres", "spheres", "hair", "glass"])
    rays = _log_int(rng, 1, 65536) if kind == "pick" else _log_int(rng, 256, 1 << 20)
    return {"kind": kind, "scene": scene, "n": n, "rays": rays, "occlusion": rng.random() < 0.4}


def _scene(case, seed):
    """The case's scene; what varies between users' scenes comes from the seed."""
    rng = np.random.default_rng(seed)
    w, h, spp, depth = (case.get(k, d) for k, d in (("width", 64), ("height", 64), ("spp", 1), ("depth", 8)))
    name, n = case["scene"], case["n"]
    if name == "cornell":
        return S.cornell(w, h, spp, depth, wall_jitter=rng.uniform(-0.1, 0.1, (3, 3)),
                         box_rot=tuple(rng.uniform(5.0, 40.0, 2) * (-1.0, 1.0)))
    if name == "spheres":
        return S.throughput(w, h, spp, depth, n_spheres=n, seed=seed)
    if name == "hair":
        return S.hair(w, h, spp, depth, n_strands=n, seed=seed)
    if name == "glass":
        return S.glass(w, h, spp, depth, seed=seed)
    if name == "motion":
        return S.motion(w, h, spp, depth, seed=seed)
    if name == "sunlit":
        return S.sunlit(w, h, spp, depth, half_angle_deg=2.0, seed=seed)
    raise ValueError(name)


def _variants(n, seed):
    """n Cornell variants in the ranges of `scenes.batched_variants`: the mix of
    sizes belongs to the case, walls and boxes to the seed."""
    size, rng = np.random.default_rng(n), np.random.default_rng(seed)
    out = []
    for _ in range(n):
        res, spp = int(size.choice([64, 128, 256, 384, 512])), int(size.choice([4, 8, 16, 32, 64]))
        out.append(S.cornell(res, res, spp, int(size.integers(4, 17)), wall_jitter=rng.uniform(-0.1, 0.1, (3, 3)),
                             box_rot=tuple(rng.uniform(5.0, 85.0, 2))))
    return out


# Where query rays start: a little beyond each scene's geometry
BOUNDS = {"cornell": (0.01, 0.99), "spheres": (-11.0, 11.0), "hair": (-1.6, 1.6), "glass": (0.2, 4.0)}


def _rays(case, sc, seed):
    """(rays, 8): origin, tmin, direction, tmax. Picks leave the camera through
    random pixels; other queries start anywhere in the scene, in any
    direction, occlusion segments with an end."""
    rng = np.random.default_rng(seed + 1)
    n = case["rays"]
    rays = np.zeros((n, 8), np.float32)
    if case["kind"] == "pick":
        at, frm = np.asarray(sc.cam_at, float), np.asarray(sc.cam_from, float)
        fwd = (at - frm) / np.linalg.norm(at - frm)
        right = np.cross(fwd, np.asarray(sc.cam_up, float))
        right /= np.linalg.norm(right)
        half = math.tan(math.radians(sc.vfov) / 2)
        xy = rng.uniform(-half, half, (n, 2))
        d = fwd + xy[:, :1] * right + xy[:, 1:] * np.cross(right, fwd)
        rays[:, 0:3] = frm
    else:
        lo, hi = BOUNDS[case["scene"]]
        rays[:, 0:3] = rng.uniform(lo, hi, (n, 3))
        d = rng.normal(0.0, 1.0, (n, 3))
    rays[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 3] = 1e-4
    rays[:, 7] = rng.uniform(0.1, 1.0, n) * (BOUNDS[case["scene"]][1] * 2.0) if case["occlusion"] else 1e10
    return rays


def prepare(case, seed):
    kind = case["kind"]
    r = api.Renderer(0)
    if kind == "batch":
        scenes = _variants(case["n"], seed)
        batch = api.Batch([api.Prepared(s) for s in scenes])
        r.upload_batch(batch)
        return {"kind": kind, "r": r, "batch": batch, "sizes": [(s.width, s.height) for s in scenes],
                "descs": [api.scene_desc_tuple(s, seed=seed) for s in scenes]}
    if kind == "gradient":
        sc = S.differentiable(case["width"], case["height"], case["spp"], case["depth"], subdiv=case["n"])
        r.upload(sc, device_build=True)
        rng = torch.Generator().manual_seed(seed)
        params = diff.initial_params(r)
        with torch.no_grad():
            params["albedo"].add_(torch.rand(params["albedo"].shape, generator=rng) * 0.1 - 0.05).clamp_(0.02, 0.95)
            params["roughness"].add_(torch.rand(params["roughness"].shape, generator=rng) * 0.1 - 0.05)
            params["roughness"].clamp_(0.05, 1.0)
        target = torch.rand((case["height"], case["width"], 3), generator=rng)
        frame = diff.Frame(case["width"], case["height"], case["spp"], case["depth"], seed=seed)
        return {"kind": kind, "r": r, "frame": frame, "params": params, "target": target}
    sc = _scene(case, seed)
    if kind == "open":
        return {"kind": kind, "r": r, "scene": sc, "case": case, "seed": seed}
    r.upload(sc, device_build=True)
    if kind == "frame":
        return {"kind": kind, "r": r, "case": case, "seed": seed}
    return {"kind": kind, "r": r, "rays": _rays(case, sc, seed), "occlusion": case["occlusion"]}


def _frame(r, c, seed):
    r.render(c["width"], c["height"], c["spp"], c["depth"], seed=seed, aovs=c["aovs"])
    film = r.film(c["width"], c["height"])
    out = {"radiance": film[..., :3], "weight": film[..., 3], "luminance2": film[..., 4]}
    if c["aovs"]:
        out["albedo"], out["normal"] = r.aovs(c["width"], c["height"])
    return out


def _hits(h):
    return {k: h[k] for k in ("hit", "mesh_id", "prim_id", "strand_id", "t", "u", "v")}


def run(state):
    kind, r = state["kind"], state["r"]
    if kind == "frame":
        return _frame(r, state["case"], state["seed"])
    if kind == "open":
        r.upload(state["scene"], device_build=True)
        return _frame(r, state["case"], state["seed"])
    if kind == "batch":
        r.render_batch(state["descs"], graph=True)
        return [r.batch_film(k, w, h) for k, (w, h) in enumerate(state["sizes"])]
    if kind == "gradient":
        p = state["params"]
        for t in p.values():
            t.grad = None
        img = diff.render(r, state["frame"], p["albedo"], p["roughness"], p["emission"], p["light_le"])
        ((img - state["target"]) ** 2).mean().backward()
        return {"image": img.detach(), **{k: t.grad for k, t in p.items()}}
    if kind == "pick":
        return _hits(r.trace_noalloc(state["rays"], occlusion=state["occlusion"]))
    return _hits(r.trace(state["rays"], occlusion=state["occlusion"]))


def _primitives(case):
    """Triangles, or curve segments where strands are the scene."""
    return {"cornell": 36, "spheres": 1280 * case["n"] + 2, "hair": 4 * case["n"], "glass": 6892, "motion": 2256,
            "sunlit": 3844, "differentiable": 36 + 20 * 4 ** case["n"]}[case["scene"]]


def work(case):
    """A ray cannot do without about two boxes per level of a binary tree and
    two primitive tests; a path without a camera ray, one shaded vertex and
    that vertex's two rays to the lights. Scene bytes are the primitives'."""
    prims = _primitives(case)
    ray = 2.0 * math.log2(prims + 1) * 18.0 + 2.0 * (300.0 if case["scene"] == "hair" else 45.0)
    scene = prims * (64.0 if case["scene"] == "hair" else 36.0)
    if case["kind"] in ("trace", "pick"):
        return {"bytes": min(scene, case["rays"] * 512.0) + 64.0 * case["rays"], "flops": case["rays"] * ray}
    if case["kind"] == "batch":
        pixels = case["n"] * 9.0e4
        return {"bytes": scene * case["n"] + 20.0 * pixels, "flops": pixels * 16.0 * (3.0 * ray + 250.0)}
    pixels = float(case["width"]) * case["height"]
    flops = pixels * case["spp"] * (3.0 * ray + 250.0)
    if case["kind"] == "gradient":  # the paths are walked forward and replayed
        return {"bytes": scene + 24.0 * pixels, "flops": 2.0 * flops}
    if case["kind"] == "open":  # vertices in, primitives and tree out
        scene *= 3.0
        flops += prims * 12.0 * math.log2(prims)
    return {"bytes": scene + (44.0 if case.get("aovs") else 20.0) * pixels, "flops": flops}


def _exact_hits(sc, rays, occlusion):
    """Nearest hit of every ray by testing every triangle, in 64 bits."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def f64(a):
        return torch.as_tensor(np.asarray(a, np.float64), device=dev)

    tri = np.asarray(sc.indices, np.int64).reshape(-1, 3)
    off = np.asarray(sc.mesh_vert_offset, np.int64)
    base = np.repeat(off[:-1], np.diff(np.asarray(sc.mesh_tri_offset, np.int64)))
    p = np.asarray(sc.positions, np.float32).reshape(-1, 3)
    v = p[tri + base[:, None]]
    v0, e1, e2 = f64(v[:, 0]), f64(v[:, 1] - v[:, 0]), f64(v[:, 2] - v[:, 0])
    n = len(rays)
    t_out, u_out, v_out = (torch.zeros(n, dtype=torch.float64, device=dev) for _ in range(3))
    step = max(1, int(2e7) // max(1, len(tri)))
    for i in range(0, n, step):
        q = f64(rays[i:i + step])
        o, d = q[:, None, 0:3], q[:, None, 4:7]
        h = torch.linalg.cross(d.expand(-1, len(tri), -1), e2[None].expand(len(q), -1, -1))
        a = (e1[None] * h).sum(-1)
        s = o - v0[None]
        u = (s * h).sum(-1) / a
        k = torch.linalg.cross(s, e1[None].expand(len(q), -1, -1))
        w = (d * k).sum(-1) / a
        t = (e2[None] * k).sum(-1) / a
        ok = (u >= 0) & (w >= 0) & (u + w <= 1) & (t >= q[:, None, 3]) & (t <= q[:, None, 7])
        t = torch.where(ok, t, torch.inf)
        best, at = t.min(1)
        hit = torch.isfinite(best)
        t_out[i:i + step] = torch.where(hit, best, 0.0)
        u_out[i:i + step] = torch.where(hit, u.gather(1, at[:, None])[:, 0], 0.0)
        v_out[i:i + step] = torch.where(hit, w.gather(1, at[:, None])[:, 0], 0.0)
    return t_out.cpu(), u_out.cpu(), v_out.cpu()


def exact(case, seed):
    """Triangle hits in 64 bits, where every triangle can be tested; a film's
    weights. A film's radiance is a Monte-Carlo estimate whose paths are chosen
    by 32-bit sample values and comparisons: no 64-bit value belongs to it,
    nor to a gradient of it."""
    if case["kind"] in ("frame", "open"):
        w = np.full((case["height"], case["width"]), float(case["spp"]))
        out = {"radiance": None, "weight": w, "luminance2": None}
        return {**out, "albedo": None, "normal": None} if case["aovs"] else out
    if case["kind"] in ("trace", "pick") and case["scene"] != "hair":
        none = {k: None for k in ("hit", "mesh_id", "prim_id", "strand_id")}
        if case["occlusion"]:  # an occlusion query answers hit alone
            zero = np.zeros(case["rays"])
            return {**none, "t": zero, "u": zero, "v": zero}
        if case["rays"] * _primitives(case) <= EXACT_TESTS:
            sc = _scene(case, seed)
            t, u, v = _exact_hits(sc, _rays(case, sc, seed), False)
            return {**none, "t": t, "u": u, "v": v}
    return None
