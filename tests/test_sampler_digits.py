"""The integer identities behind the device sampler's digits
(csrc/sampler.cuh): the later digits' 32-bit reciprocal and the closed form of
the base-2 radical inverse, against the digit loop in single precision."""
import numpy as np

from tests.test_sampler_tables import _primes


def test_later_digits_by_32_bit_reciprocal():
    rng = np.random.default_rng(1)
    for b in _primes(128):
        magic = -(-(1 << 64) // b)
        m = (magic >> 32) + (1 if b > 2 else 0)
        assert m == -(-(1 << 32) // b) and m < 1 << 32
        top = ((1 << 32) - 1) // b  # the largest quotient a first digit leaves
        ns = [0, 1, b - 1, b, b + 1, *range(top - 2 * b, top + 1), *map(int, rng.integers(0, top + 1, 500))]
        for n in ns:
            assert (n * m) >> 32 == n // b
        for n in [0, b - 1, b, (1 << 32) - 1, (1 << 32) - b, *map(int, rng.integers(0, 1 << 32, 200))]:
            assert (n * (magic >> 32) + ((n * (magic & 0xFFFFFFFF)) >> 32)) >> 32 == n // b


def test_base_two_closed_form():
    rng = np.random.default_rng(2)
    n = np.concatenate([np.arange(1 << 12), (1 << 32) - 1 - np.arange(1 << 12), 1 << np.arange(32),
                        (1 << 32) - (1 << np.arange(32)), rng.integers(0, 1 << 32, 200_000)]).astype(np.uint64)
    r, w, left = np.zeros(len(n), np.float32), np.float32(1.0), n.copy()
    for _ in range(32):
        w = w * np.float32(0.5)
        r = r + (left & np.uint64(1)).astype(np.float32) * w
        left >>= np.uint64(1)
    v = np.zeros_like(n)
    for i in range(32):
        v |= ((n >> np.uint64(i)) & np.uint64(1)) << np.uint64(31 - i)
    lz = np.array([32 - max(1, int(x)).bit_length() for x in v], np.uint64)
    cut = v & (np.uint64(0xFFFFFF80) >> lz)
    assert np.array_equal(cut.astype(np.float32) * np.float32(2.0 ** -32), r)
