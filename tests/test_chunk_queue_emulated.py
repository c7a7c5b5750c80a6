"""The chunk dictionary's hash and its warps' key queues (fls_cd_queue.cuh) on the CPU: keys that crowd on one place
spend a warp's looks without ever outgrowing the queue."""
import ctypes

import numpy as np
import pytest

from tests import chunk_keys as CK
from tests.emu import build


@pytest.fixture(scope="module")
def emu():
    return ctypes.CDLL(build.build())


def P(a):
    return ctypes.c_void_p(a.ctypes.data)


def _hash(emu, keys):
    place, other = np.zeros(keys.size, np.uint32), np.zeros(keys.size, np.uint32)
    emu.emu_cd_hash(8 * keys.itemsize, P(keys), ctypes.c_uint64(keys.size), P(place), P(other))
    return place, other


def test_hash_is_the_one_the_tests_invert(emu):
    rng = np.random.default_rng(1)
    place = rng.integers(0, 2**32, 4096, dtype=np.uint64).astype(np.uint32)
    other = rng.integers(0, 2**32, 4096, dtype=np.uint64).astype(np.uint32)
    p, o = _hash(emu, np.ascontiguousarray(CK.key64(place, other)))
    assert np.array_equal(p, place) and np.array_equal(o, other)
    p, o = _hash(emu, np.ascontiguousarray(CK.key32(place)))
    assert np.array_equal(p, place) and np.array_equal(o, place << np.uint32(16))


@pytest.mark.parametrize("a,b", [(56, 24), (32, 0), (48, 16), (40, 20), (33, 31)])
def test_structured_keys_spread(emu, a, b):
    """Keys of two 8-bit fields (65,536 of them, fewer where the fields overlap): they take as many of the table's 47 Ki
    slots as random keys do, m (1 - exp(-n / m)) with a standard deviation below sqrt(n), and half of them each part."""
    i = np.arange(65536, dtype=np.uint64)
    keys = np.unique(((i >> np.uint64(8)) << np.uint64(a)) + ((i & np.uint64(255)) << np.uint64(b)))
    place, other = _hash(emu, keys)
    n, m = keys.size, 47 * 1024
    slots = np.unique((place.astype(np.uint64) * np.uint64(m)) >> np.uint64(32)).size
    assert slots > m * (1 - np.exp(-n / m)) - 4 * np.sqrt(n)
    part = (other >> np.uint32(16)) & np.uint32(1)
    assert abs(int(part.sum()) - n / 2) < 4 * np.sqrt(n)


@pytest.mark.parametrize("n_slots,looks,crowd", [(2048, 1 << 14, False), (2048, 1 << 14, True), (2048, 100, True),
                                                 (2048, 1, True), (2048, 0, True)])
def test_queue_is_never_outgrown(emu, n_slots, looks, crowd):
    """32 rows of 32 different keys, a third of them held back, spread or all on one place, with enough looks and with
    too few."""
    rng = np.random.default_rng(looks + crowd)
    n = 1024
    keys = np.ascontiguousarray(CK.key64(5 if crowd else rng.integers(0, 2**32, n, dtype=np.uint64), np.arange(n)))
    need = (rng.random(n) < 0.7).astype(np.uint8)
    fresh = ctypes.c_uint32()
    got = emu.emu_cd_queue(P(keys), P(need), 32, n_slots, looks, ctypes.byref(fresh))
    if looks == 1 << 14:
        assert 32 <= got <= 64 and fresh.value == int(need.sum())
    else:
        assert got == -1  # the looks were spent, and nothing written outside the queue
