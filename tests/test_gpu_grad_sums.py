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
