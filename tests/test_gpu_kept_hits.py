"""Kept hits of the backward pass on the device."""
import numpy as np
import pytest

from anacapa_b200 import api
from anacapa_b200 import scenes as S

pytestmark = pytest.mark.gpu


def test_room_with_other_scenes_hits(gpu):
    """A context whose room for hits was filled by deeper passes over a larger
    scene gives the gradients of a fresh one (up to the order of the
    single-precision atomic sums)."""
    small = S.differentiable(96, 64, 4, 12, subdiv=1)
    d = np.random.default_rng(4).normal(size=(64, 96, 3)).astype(np.float32) / (96 * 64)
    used, fresh = api.Renderer(chunk_paths=5000), api.Renderer(chunk_paths=5000)
    try:
        used.upload(S.differentiable(96, 64, 4, 16, subdiv=5))
        used.forward(96, 64, 4, 16)
        used.backward(d)
        out = []
        for r in (used, fresh):
            r.upload(small)
            r.forward(96, 64, 4, 12)
            out.append(r.backward(d))
        for k in out[0]:
            a, b = out[0][k].astype(np.float64), out[1][k].astype(np.float64)
            assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b) + 1e-12, k
    finally:
        used.close()
        fresh.close()
