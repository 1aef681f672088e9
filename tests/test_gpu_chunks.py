"""The default chunk around 2^25 paths: one chunk up to there, 2^26 paths for a
larger frame; films do not depend on where chunks are cut."""
import numpy as np
import pytest

from anacapa_b200 import api
from anacapa_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp,default,fixed", [(2048, 1024, 16, 1, 1), (2049, 1024, 16, 1, 2),
                                                   (2048, 1025, 33, 2, 3)])
def test_default_chunks(gpu, w, h, spp, default, fixed):
    sc = S.sunlit(w, h, spp, 1)
    films = []
    for chunk, want in ((0, default), (1 << 25, fixed)):
        r = api.Renderer(chunk_paths=chunk)
        try:
            r.upload(sc)
            r.render_scene(sc)
            assert r.stats().chunks == want
            films.append(r.film(w, h))
        finally:
            r.close()
    assert np.array_equal(*films)
