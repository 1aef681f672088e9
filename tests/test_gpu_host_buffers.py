"""Films, AOVs, gradients' images and queries in page-locked buffers, which the
driver moves directly, against pageable ones, which cross in pinned chunks of
128 KiB dealt to four threads: sizes at a chunk's and at a round's end."""
import numpy as np
import pytest

from anacapa_b200 import api
from anacapa_b200 import scenes as S
from tests.test_gpu_queue_edges import random_rays

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CHUNK, ROUND = 1 << 17, 4 << 17


def _locked(shape):
    return torch.zeros(shape, dtype=torch.float32, pin_memory=True)


# pixels of 20 bytes (AOVs 12): multiples of 128 KiB and 512 KiB above 1 MiB, and one pixel to both sides
PIXELS = sorted({max(1, -(-k * b // z)) + e for b in (CHUNK, ROUND) for k in (8, 9, 13) for z in (20, 12)
                 for e in (-1, 0, 1)})


@pytest.mark.parametrize("pixels", PIXELS)
def test_films_and_aovs(gpu, pixels):
    w, h = (pixels, 1) if pixels < 1 << 16 else (pixels // 4, 4)
    n = w * h
    sc = S.sunlit(w, h, 1, 2)
    r = api.Renderer()
    try:
        r.upload(sc)
        r.render_scene(sc, aovs=True)
        film = _locked((h, w, 5))
        api.check(api.lib().ana_film_read(r.h, film.data_ptr(), n), r.h)
        assert np.array_equal(film.numpy(), r.film(w, h))
        assert (film[..., 3] == 1).all() and (film[..., :3] > 0).any()
        al, nr = _locked((h, w, 3)), _locked((h, w, 3))
        api.check(api.lib().ana_aov_read(r.h, al.data_ptr(), nr.data_ptr(), n), r.h)
        got = r.aovs(w, h)
        assert np.array_equal(al.numpy(), got[0]) and np.array_equal(nr.numpy(), got[1])
        assert (al > 0).any() and (nr != 0).any()
    finally:
        r.close()


@pytest.mark.parametrize("occlusion", [0, 1])
def test_queries(gpu, occlusion):
    sc = S.throughput(64, 36, 1, 4, n_spheres=48, subdiv=2)
    r = api.Renderer()
    try:
        r.upload(sc)
        for n in (ROUND // 16 - 1, ROUND // 16, ROUND // 16 + 1, 9 * CHUNK // 32 + 1, 5 * ROUND // 32 - 1):
            rays = random_rays(n, 11.0, n)
            locked, out = torch.from_numpy(rays).pin_memory(), _locked((n, 8))
            api.check(api.lib().ana_trace_batch(r.h, locked.data_ptr(), n, out.data_ptr(), occlusion, 0), r.h)
            assert out.numpy().tobytes() == r.trace(rays, occlusion=bool(occlusion)).tobytes()
    finally:
        r.close()


def test_forward_image_and_gradient_image(gpu):
    w, h, spp, depth = 320, 300, 2, 3
    sc = S.differentiable(w, h, spp, depth, subdiv=2)
    d = np.random.default_rng(8).normal(size=(h, w, 3)).astype(np.float32) / (w * h)
    r = api.Renderer()
    try:
        r.upload(sc)
        img = r.forward(w, h, spp, depth)
        a = r.backward(d)
        locked = torch.from_numpy(d).pin_memory()
        b = r.backward(locked.numpy())
        for k in a:
            assert np.linalg.norm(a[k] - b[k]) <= 1e-4 * np.linalg.norm(a[k]) + 1e-12, k
        film = r.film(w, h)
        assert np.array_equal(img, film[..., :3] / film[..., 3:4])
    finally:
        r.close()


def test_copies_after_a_set_has_taken_larger_chunks(gpu):
    """1 MiB chunks from 128 MiB on: films around their ends and their rounds'."""
    r = api.Renderer()
    try:
        r.upload(S.sunlit(64, 64, 1, 2))
        r.render(1920, 1080, 1, 1)
        for _ in range(4):  # 41 MB each
            r.film(1920, 1080)
        for mib in (1, 2, 4, 5, 8, 13):
            for e in (-1, 0, 1):
                w = -(-(mib << 20) // 20) + e
                r.render(w, 1, 1, 1)
                film = _locked((1, w, 5))
                api.check(api.lib().ana_film_read(r.h, film.data_ptr(), w), r.h)
                assert np.array_equal(film.numpy(), r.film(w, 1))
        rays = random_rays(9 * (1 << 15) + 5, 11.0, 3)
        locked, out = torch.from_numpy(rays).pin_memory(), _locked((len(rays), 8))
        api.check(api.lib().ana_trace_batch(r.h, locked.data_ptr(), len(rays), out.data_ptr(), 0, 0), r.h)
        assert out.numpy().tobytes() == r.trace(rays).tobytes()
    finally:
        r.close()
