"""Copies around the sizes where the host path changes (1024 rays, 1 MiB, the
pinned chunks' 1 MiB multiples): queries and films against the same work read in
other sizes, two contexts on two threads at once, and the AOV and image
resolves against the host's arithmetic on the same film."""
import threading

import numpy as np
import pytest

from anacapa_b200 import api
from anacapa_b200 import scenes as S
from tests.test_gpu_queue_edges import random_rays

pytestmark = pytest.mark.gpu

RAYS = [1, 1023, 1024, 1025, 32767, 32768, 32769, 65536, 5 * 32768 + 3, 9 * 32768 + 1]


@pytest.mark.parametrize("occlusion", [False, True])
def test_query_sizes(gpu, occlusion):
    sc = S.throughput(64, 36, 1, 4, n_spheres=48, subdiv=2)
    r = api.Renderer()
    try:
        r.upload(sc)
        rays = random_rays(max(RAYS), 11.0, 31)
        rays[:, 7] = 4.0
        want = np.concatenate([r.trace(rays[i:i + 900], occlusion=occlusion) for i in range(0, len(rays), 900)])
        assert 0 < want["hit"].sum() < len(want)
        for n in RAYS:
            assert np.array_equal(r.trace(rays[:n], occlusion=occlusion), want[:n])
            assert np.array_equal(r.trace(rays[:n], occlusion=occlusion, times=np.zeros(n)), want[:n])
            if n <= api.TRACE_NOALLOC_MAX_RAYS:
                assert np.array_equal(r.trace_noalloc(rays[:n], occlusion=occlusion), want[:n])
    finally:
        r.close()


@pytest.mark.parametrize("size", [(229, 229), (229, 228), (512, 102), (1000, 524), (1024, 1024)])
def test_films_and_resolves(gpu, size):
    """20-byte pixels: films just under and over 1 MiB, a ragged last chunk."""
    w, h = size
    sc = S.sunlit(w, h, 1, 2)
    r = api.Renderer()
    try:
        r.upload(sc)
        r.render_scene(sc, aovs=True)
        f = r.film(w, h)
        assert np.array_equal(f[..., 3], np.ones((h, w), np.float32))
        rows = np.concatenate([t[None] for t in f])  # a second read is the same
        assert np.array_equal(rows, r.film(w, h))
        al, nr = r.aovs(w, h)
        assert np.isfinite(al).all() and np.isfinite(nr).all() and (al > 0).any()
        hit = (nr != 0).any(-1)
        assert np.allclose(np.linalg.norm(nr[hit].astype(np.float64), axis=1), 1.0, atol=1e-5)
        img = r.forward(w, h, 1, 2)
        f = r.film(w, h)
        assert np.array_equal(img, f[..., :3] / f[..., 3:4])
    finally:
        r.close()


def test_two_contexts_on_two_threads(gpu):
    sc = S.sunlit(640, 480, 1, 3)
    rs = [api.Renderer() for _ in range(2)]
    try:
        for r in rs:
            r.upload(sc)
            r.render_scene(sc)
        want = rs[0].film(640, 480)
        rays = random_rays(200_003, 4.0, 32)
        hits = rs[0].trace(rays)
        bad = []

        def work(r):
            for _ in range(6):
                if not (np.array_equal(r.film(640, 480), want) and np.array_equal(r.trace(rays), hits)):
                    bad.append(r)

        ts = [threading.Thread(target=work, args=(r,)) for r in rs]
        [t.start() for t in ts]
        [t.join() for t in ts]
        assert not bad
    finally:
        [r.close() for r in rs]
