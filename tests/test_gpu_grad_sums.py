"""Gradient sums of warps whose lanes hold few, many and no parameters: films
around a warp's 32 paths, against the FP64 adjoint of the same paths (the bar
of the adjoint tests)."""
import numpy as np
import pytest

from anacapa_b200 import api
from anacapa_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1, 1), (31, 1, 1), (4, 8, 1), (11, 3, 1), (40, 24, 3)])
def test_small_films_match_fp64_adjoint(gpu, restate_built, size):
    w, h, spp = size
    sc = S.differentiable(w, h, spp, 3, subdiv=2)
    r = api.Renderer()
    try:
        r.upload(sc)
        r.forward(w, h, spp, 3)
        d = np.random.default_rng(w).normal(size=(h, w, 3)).astype(np.float32)
        g = r.backward(d)
        nm, nl = r.diff_counts()
        got = np.zeros(8 * nm + 4 * nl)
        for i in range(nm):
            got[8 * i:8 * i + 3], got[8 * i + 3] = g["albedo"][i], g["roughness"][i]
            got[8 * i + 4:8 * i + 7] = g["emission"][i]
        for i in range(nl):
            got[8 * nm + 4 * i:8 * nm + 4 * i + 3] = g["light_le"][i]
        ref = restate_built.PoScene(sc, precision=64).adjoint(d)
        assert np.linalg.norm(got - ref) <= 1e-3 * max(np.linalg.norm(ref), 1e-30)
    finally:
        r.close()


def test_kept_hits_and_traced_hits_agree(gpu):
    """The adjoint replay takes the primal's hits while they fit the room for
    them: a chunk of 2^20 paths fits at any depth up to 255, one of 2^22 at
    depth 255 does not and is traced again. Same paths, same gradient up to the
    order of its single-precision atomic sums."""
    w, h, spp = 512, 512, 16
    sc = S.differentiable(w, h, spp, 255, subdiv=2)
    d = np.random.default_rng(3).normal(size=(h, w, 3)).astype(np.float32) / (w * h)
    out = []
    for chunk in (1 << 20, 1 << 22):
        r = api.Renderer(chunk_paths=chunk)
        try:
            r.upload(sc)
            r.forward(w, h, spp, 255)
            out.append(r.backward(d))
        finally:
            r.close()
    for k in out[0]:
        a, b = out[0][k].astype(np.float64), out[1][k].astype(np.float64)
        assert np.linalg.norm(a - b) <= 1e-3 * np.linalg.norm(b) + 1e-12, k


def test_kept_curve_hits(gpu, restate_built):
    """Curve hits carry a second record; hair is not differentiated, the quad's
    light is, through paths that meet strands."""
    sc = S.hair(48, 32, 2, 4, n_strands=2000)
    r = api.Renderer()
    try:
        r.upload(sc)
        r.forward(48, 32, 2, 4)
        d = np.random.default_rng(5).normal(size=(32, 48, 3)).astype(np.float32)
        g = r.backward(d)
        ref = restate_built.PoScene(sc, precision=64).adjoint(d)
        nm = len(sc.materials)
        got, want = g["light_le"][0], ref[8 * nm:8 * nm + 3]
        assert np.linalg.norm(got - want) <= 1e-3 * np.linalg.norm(want)
    finally:
        r.close()
