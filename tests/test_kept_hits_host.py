"""The hits that the primal replay of a backward pass keeps for the adjoint
replay, on the host side of the library."""
from contextlib import closing

import numpy as np
import pytest

from anacapa_b200 import api
from anacapa_b200 import scenes as S
from tests.fake_device import fake_device


@pytest.mark.parametrize("curves", [False, True])
@pytest.mark.parametrize("chunk", [0, 1000, 4096])
def test_paths_the_primal_did_not_walk_have_no_hit(chunk, curves):
    """The room for the hits holds whatever was there before. Where the adjoint
    replay comes to a bounce that its path did not reach in the primal replay
    (two kernels, whose roulette may round differently), it finds that said, in
    every chunk, and not a primitive index from older memory."""
    w, h, spp, depth = 40, 30, 4, 5
    sc = S.hair(w, h, spp, depth, n_strands=50) if curves else S.differentiable(w, h, spp, depth, subdiv=1)
    with fake_device() as L, closing(api.Renderer(chunk_paths=chunk)) as r:
        r.upload(sc)
        for _ in range(2):
            r.forward(w, h, spp, depth)
            r.backward(np.ones((h, w, 3), np.float32))
        assert L.fake_good_records() == 2 * w * h * spp * (depth + 1)
        assert L.fake_bad_records() == 0
