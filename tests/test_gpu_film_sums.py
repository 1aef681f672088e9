"""Film sums around the tiles of samples and the warps of pixels: every film
equals the sum of passes of one sample each, which are summed in the same order
pass by pass, and batches whose scenes change inside a warp equal their scenes
rendered alone."""
import numpy as np
import pytest

from anacapa_b200 import api
from anacapa_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spp", [1, 7, 15, 16, 17, 31, 32, 33, 64])
def test_samples_per_pixel(gpu, spp):
    """33 x 5 pixels (a ragged warp). One-sample passes add each sample's
    radiance to the film, the frame adds its mean times spp: equal up to that
    division's rounding (2 of 2^-24 per channel, plus one per addition)."""
    w, h = 33, 5
    sc = S.sunlit(w, h, spp, 3)
    r = api.Renderer()
    try:
        r.upload(sc)
        for k in range(spp):
            r.render(w, h, 1, 3, sample_start=k, clear=k == 0, aovs=True)
        one = r.film(w, h)
        al1, nr1 = r.aovs(w, h)
        r.render(w, h, spp, 3, aovs=True)
        f = r.film(w, h)
        al, nr = r.aovs(w, h)
        assert np.array_equal(f[..., 3], one[..., 3])
        tol = (spp + 4) * 2.0 ** -24
        assert np.allclose(f[..., :3], one[..., :3], rtol=tol, atol=0)
        assert np.allclose(f[..., 4], one[..., 4], rtol=2 * tol, atol=0)
        # an AOV pass stores its albedo mean, averaged over the passes
        assert np.allclose(al, al1, rtol=2 * tol, atol=1e-7)
        if spp == 1:
            assert np.array_equal(nr, nr1)
    finally:
        r.close()


def test_scenes_meeting_inside_a_warp(gpu):
    scs = [S.cornell(w, h, spp, 3) for w, h, spp in [(5, 3, 32), (7, 1, 33), (1, 1, 40), (33, 1, 1), (9, 9, 48)]]
    r = api.Renderer()
    try:
        alone = []
        for sc in scs:
            r.upload(sc)
            r.render_scene(sc)
            alone.append(r.film(sc.width, sc.height))
        r.upload_batch(api.Batch([api.Prepared(sc) for sc in scs]))
        r.render_batch([api.scene_desc_tuple(sc) for sc in scs])
        for k, sc in enumerate(scs):
            assert np.array_equal(r.batch_film(k, sc.width, sc.height), alone[k])
    finally:
        r.close()
