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


W, H, SPP, DEPTH = 40, 30, 4, 5
ROOM = -(-W * H * SPP * 16 // 256) * 256 * (DEPTH + 1)


def _backward(r, w=W, h=H):
    r.forward(w, h, SPP, DEPTH)
    r.backward(np.ones((h, w, 3), np.float32))


def _held_without_hits(sc):
    with fake_device() as L, closing(api.Renderer()) as r:
        L.fake_fail(b"cudaMemGetInfo", 0, -1)
        r.upload(sc)
        _backward(r)
        assert L.fake_good_records() == 0
        return L.fake_held()


def test_hits_are_kept_in_a_part_of_free_memory():
    """Room for them is taken only where it is a sixteenth of what is free, and
    the pass does without it where it is not, or cannot be had."""
    sc = S.differentiable(W, H, SPP, DEPTH, subdiv=1)
    other = _held_without_hits(sc)
    for free, kept in ((16 * ROOM, True), (16 * ROOM - 16, False)):
        with fake_device(capacity=other + free) as L, closing(api.Renderer()) as r:
            r.upload(sc)
            _backward(r)
            assert (L.fake_good_records() > 0) == kept
            assert L.fake_held() == other + (ROOM if kept else 0)
    with fake_device() as L, closing(api.Renderer()) as r:
        r.upload(sc)
        r.forward(W, H, SPP, DEPTH)
        # queues, image, counters of the pass come first; the last one is the room
        L.fake_fail(b"cudaMalloc", 3, 1)
        r.backward(np.ones((H, W, 3), np.float32))
        assert L.fake_good_records() == 0 and L.fake_held() == other


def test_room_for_hits_is_given_back():
    sc = S.differentiable(W, H, SPP, DEPTH, subdiv=1)
    other = _held_without_hits(sc)
    with fake_device() as L, closing(api.Renderer()) as r:
        r.upload(sc)
        for _ in range(3):
            _backward(r)
            assert L.fake_held() == other + ROOM
        allocations = L.fake_calls(b"cudaMalloc")
        _backward(r)
        assert L.fake_calls(b"cudaMalloc") == allocations
        _backward(r, 20, 10)  # a smaller frame: less than half of it
        assert L.fake_held() - other < ROOM // 4
        _backward(r)
        r.upload(sc)
        assert L.fake_held() == other
        _backward(r)
        r.trace(np.ones((4, 8), np.float32))  # its own buffer
        assert L.fake_held() > other + ROOM


def test_other_allocations_come_before_the_room_for_hits():
    sc = S.differentiable(W, H, SPP, DEPTH, subdiv=1)
    with fake_device() as L, closing(api.Renderer()) as r:
        r.upload(sc)
        _backward(r)
        held = L.fake_held()
        L.fake_fail(b"cudaMalloc", 0, 1)
        out = r.trace(np.full((5000, 8), 3.0, np.float32))
        assert (out["t"] == 3).all()
        assert L.fake_held() < held


@pytest.mark.parametrize("kept", [True, False])
def test_statistics_count_the_rays_that_are_traced(kept):
    sc = S.differentiable(W, H, SPP, DEPTH, subdiv=1)
    with fake_device() as L, closing(api.Renderer(chunk_paths=1000)) as r:
        if not kept:
            L.fake_fail(b"cudaMemGetInfo", 0, -1)
        r.upload(sc)
        r.forward(W, H, SPP, DEPTH)
        forward = L.fake_extend_rays()
        assert r.stats().extend_rays == forward > 0
        r.backward(np.ones((H, W, 3), np.float32))
        assert r.stats().extend_rays == L.fake_extend_rays() - forward == (1 if kept else 2) * forward
        assert r.stats().bounces == DEPTH + 1
