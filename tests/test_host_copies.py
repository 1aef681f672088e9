"""Copies between host memory and the device: which route a buffer takes."""
from contextlib import ExitStack, closing

import numpy as np
import pytest

from anacapa_b200 import api
from anacapa_b200 import scenes as S
from tests.fake_device import DEVICE, HOST, MANAGED, fake_device

W, H = 320, 240  # films of 1.5 MB


def _rendered(r):
    sc = S.cornell(W, H, 1, 2)
    r.upload(sc)
    r.render(W, H, 1, 2)


def _film(L, r, kind):
    out = np.empty((H, W, 5), np.float32)
    if kind is not None:
        L.fake_mark(out.ctypes.data, out.nbytes, kind)
    before, chunks = L.fake_direct_bytes(), L.fake_calls(b"cudaEventSynchronize")
    api.check(L.ana_film_read(r.h, out.ctypes.data, W * H), r.h)
    L.fake_mark(out.ctypes.data, 0, -1)
    assert np.array_equal(out[..., 0].ravel(), np.arange(W * H, dtype=np.float32))
    return L.fake_direct_bytes() - before, L.fake_calls(b"cudaEventSynchronize") - chunks


@pytest.mark.parametrize("kind", [HOST, MANAGED, DEVICE])
def test_memory_that_the_driver_moves_directly_is_left_to_it(kind):
    with fake_device() as L, closing(api.Renderer()) as r:
        _rendered(r)
        assert _film(L, r, kind) == (W * H * 20, 0)
        assert _film(L, r, None)[0] == 0  # pageable: through the pinned chunks


def test_page_locked_queries():
    n = 70_000
    rays, out = np.random.default_rng(0).random((n, 8), np.float32), np.zeros(n, api.HIT_DTYPE)
    with fake_device() as L, closing(api.Renderer()) as r:
        _rendered(r)
        before = L.fake_direct_bytes()
        api.check(L.ana_trace_batch(r.h, rays.ctypes.data, n, out.ctypes.data, 0, 0), r.h)
        pageable = L.fake_direct_bytes() - before
        for a in (rays, out):
            L.fake_mark(a.ctypes.data, a.nbytes, HOST)
        want, out[:] = out.copy(), np.zeros((), api.HIT_DTYPE)
        api.check(L.ana_trace_batch(r.h, rays.ctypes.data, n, out.ctypes.data, 0, 0), r.h)
        assert L.fake_direct_bytes() - before - 2 * pageable == 2 * 32 * n
        assert np.array_equal(out, want) and np.array_equal(out["t"], rays[:, 0])
        # of the rays only the first half is page-locked: none is assumed to be
        L.fake_mark(rays.ctypes.data, rays.nbytes // 2, HOST)
        before = L.fake_direct_bytes()
        api.check(L.ana_trace_batch(r.h, rays.ctypes.data, n, out.ctypes.data, 0, 0), r.h)
        assert L.fake_direct_bytes() - before - pageable == 32 * n  # the hits
        for a in (rays, out):
            L.fake_mark(a.ctypes.data, 0, -1)


def test_a_failed_query_leaves_no_copy_of_the_callers_memory_running():
    n = 70_000
    rays, out = np.ones((n, 8), np.float32), np.zeros(n, api.HIT_DTYPE)
    with fake_device() as L, closing(api.Renderer()) as r:
        _rendered(r)
        for a in (rays, out):
            L.fake_mark(a.ctypes.data, a.nbytes, HOST)
        waits = L.fake_calls(b"cudaStreamSynchronize")
        L.fake_fail(b"cudaMemcpyAsync", 2, 1)  # after the scene record and the rays: the hits
        assert L.ana_trace_batch(r.h, rays.ctypes.data, n, out.ctypes.data, 0, 0) == api.ANA_ERR_CUDA
        assert L.fake_calls(b"cudaStreamSynchronize") == waits + 1
        api.check(L.ana_trace_batch(r.h, rays.ctypes.data, n, out.ctypes.data, 0, 0), r.h)
        assert (out["t"] == 1).all()
        for a in (rays, out):
            L.fake_mark(a.ctypes.data, 0, -1)


@pytest.mark.parametrize("size", [(W, H), (129, 127), (1, 1)])
def test_images_resolve_without_device_memory(size):
    """A device without room for a resolved image: the same pixels."""
    w, h = size
    sc = S.differentiable(w, h, 1, 2, subdiv=1)
    images = []
    with fake_device() as L:
        for full in (False, True):
            with closing(api.Renderer()) as r:
                r.upload(sc)
                r.render(w, h, 1, 2, aovs=True)
                held = L.fake_held()
                if full:
                    L.fake_fail(b"cudaMalloc", 0, -1)
                images.append([*r.aovs(w, h), r.forward(w, h, 1, 2)])
                assert (L.fake_held() == held) == full
    for a, b in zip(*images):
        assert np.array_equal(a, b)
    al, nr, img = images[1]
    i = np.arange(w * h, dtype=np.float32)
    assert np.array_equal(al[..., 0].ravel(), i / 4) and (nr == 0).all()
    assert np.array_equal(img[..., 2].ravel(), 3 * i / 2)


def test_idle_sets_are_kept_by_device():
    """Contexts on four devices, whose copies alternate: no set is made twice,
    a device's sets go with its last context, and page-locked memory with them."""
    with fake_device() as L, ExitStack() as stack:
        rs = [stack.enter_context(closing(api.Renderer(device=d))) for d in (0, 1, 2, 3, 3)]
        for r in rs:
            _rendered(r)
            r.film(W, H)
        made = L.fake_calls(b"cudaHostAlloc")
        for _ in range(3):
            for r in rs:
                r.film(W, H)
        assert L.fake_calls(b"cudaHostAlloc") == made
        freed = L.fake_calls(b"cudaStreamDestroy")
        rs.pop().close()  # the fourth device has another context
        assert L.fake_calls(b"cudaStreamDestroy") == freed + 2  # its own two
        rs.pop().close()
        assert L.fake_calls(b"cudaStreamDestroy") > freed + 4
        again = stack.enter_context(closing(api.Renderer(device=3)))
        _rendered(again)
        made = L.fake_calls(b"cudaHostAlloc")
        again.film(W, H)
        assert L.fake_calls(b"cudaHostAlloc") == made + 1


@pytest.mark.parametrize("threads", [0, 1, 2])
def test_a_copy_without_memory_for_its_threads(threads):
    """The calling thread copies the part of those that could not be started."""
    with fake_device() as L, closing(api.Renderer()) as r:
        _rendered(r)
        want = r.film(W, H)
        out = np.zeros_like(want)
        L.fake_fail_new(threads)
        rc = L.ana_film_read(r.h, out.ctypes.data, W * H)
        L.fake_fail_new(-1)
        assert rc == api.ANA_OK and np.array_equal(out, want)


def test_sets_in_steady_use_take_larger_chunks():
    """Once, after 128 MiB; without page-locked memory for them the small ones
    stay in use, and are not given up."""
    per = W * H * 20
    reads = -(-(128 << 20) // per)
    for refused in (False, True):
        with fake_device() as L, closing(api.Renderer()) as r:
            _rendered(r)
            want = r.film(W, H)
            made = L.fake_calls(b"cudaHostAlloc")
            for _ in range(reads - 1):
                r.film(W, H)
            assert L.fake_calls(b"cudaHostAlloc") == made
            waits = L.fake_calls(b"cudaEventSynchronize")
            if refused:
                L.fake_fail(b"cudaHostAlloc", 0, 1)
            assert np.array_equal(r.film(W, H), want)
            chunk = (1 << 17) if refused else (1 << 20)
            assert L.fake_calls(b"cudaEventSynchronize") - waits == -(-per // chunk)
            assert L.fake_calls(b"cudaHostAlloc") == made + 1
            for _ in range(3):
                assert np.array_equal(r.film(W, H), want)
            assert L.fake_calls(b"cudaHostAlloc") == made + 1
