"""Which columns of a string set its CTAs take (fls_strings.cuh), on the CPU: CTAs that ask together spread over columns that
have equally much left, the fullest one wins otherwise, and a finished set has none."""
import ctypes

import numpy as np

from tests.emu import build


def _columns(n_vec, taken, ctas):
    emu = ctypes.CDLL(build.build())
    first = np.concatenate([[0], np.cumsum(n_vec)]).astype(np.uint64)
    flags = np.concatenate([[0], taken]).astype(np.uint64)
    share, fullest = np.zeros(ctas, np.uint32), np.zeros(ctas, np.uint32)
    P = lambda a: ctypes.c_void_p(a.ctypes.data)
    emu.emu_set_columns(P(first), P(flags), len(n_vec), ctas, P(share), P(fullest))
    return share.tolist(), fullest.tolist()


def test_columns_of_equal_size_are_spread():
    for n in (7, 60, 148, 300):
        share, fullest = _columns([64] * n, [10] * n, 148)
        assert len(set(fullest)) == min(n, 148) and len(set(share)) == min(n, 148)


def test_the_fullest_column_is_taken():
    share, fullest = _columns([5, 100, 5, 60], [0, 90, 6, 0], 20)
    assert fullest == [3] * 20
    assert [share.count(c) for c in range(4)] == [1, 12, 0, 7]


def test_nothing_left():
    assert _columns([3, 64, 1], [3, 70, 1], 5)[1] == [3] * 5
