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


def test_statistics_tell_kept_from_traced_hits(gpu):
    """The two routes of the adjoint replay, told apart by the rays they trace,
    give the same gradient. 2^14 paths to depth 24 fit the room for hits; the
    same frame to depth 255 in one chunk of 2^21 paths does not."""
    d = np.random.default_rng(6).normal(size=(128, 128, 3)).astype(np.float32) / (128 * 128)
    for (w, h, spp), depth, kept in (((128, 128, 1), 24, True), ((512, 512, 8), 255, False)):
        sc = S.differentiable(w, h, spp, depth, subdiv=2)
        out = []
        for chunk in (1 << 21, 1 << 12 if kept else 1 << 16):
            r = api.Renderer(chunk_paths=chunk)
            try:
                r.upload(sc)
                r.forward(w, h, spp, depth)
                forward = r.stats().extend_rays
                g = r.backward(np.resize(d, (h, w, 3)))
                traced = r.stats().extend_rays / forward
                if kept or chunk < 1 << 21:
                    assert traced == 1
                else:
                    assert 1.99 < traced < 2.01
                out.append(g)
            finally:
                r.close()
        for k in out[0]:
            a, b = out[0][k].astype(np.float64), out[1][k].astype(np.float64)
            assert np.linalg.norm(a - b) <= 1e-3 * np.linalg.norm(b) + 1e-12, k
