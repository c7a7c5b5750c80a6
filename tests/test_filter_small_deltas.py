"""Predicates on DELTA pages of 64-bit keys with small gaps (the filter's 32-bit range test on the running sums):
every operator at constants on and beside chain starts and ends, outside the values, and at the type's limits, for
columns that cross zero, the middle and the end of the 64-bit range, signed and unsigned; and the index lists of
empty, full and ragged bitmaps at every alignment of the output."""
import ctypes

import numpy as np
import pytest

from oracle import oracle
from oracle import predicate as PR
from tests.emu import build

STARTS = (0, -5000, 2**63 - 4000, -(2**63), 2**64 - 3000, 10**18)


def _values(start, max_gap):
    rng = np.random.default_rng(abs(start) % 1000 + max_gap)
    gaps = rng.integers(0, max_gap + 1, 2 * 1024, dtype=np.uint64)
    return np.uint64(start % 2**64) + np.cumsum(gaps, dtype=np.uint64)


def _delta_page(u):
    """DELTA_NO_PATCH page (include/fls/cor/exp/delta/delta_exp.hpp:39-56): lane bases, widths, bases, packed."""
    lanes, bws, bases, packed, ep = b"", b"", b"", b"", []
    for v in range(u.size // 1024):
        tr = oracle.transpose_i(u[v * 1024:(v + 1) * 1024].copy())
        d = oracle.unrsum(tr)
        bw, base = int(d.max() - d.min()).bit_length(), int(d.min())
        ep.append([len(lanes), len(bws), len(bases), len(packed)])
        lanes += tr[:16].tobytes()
        bws += bytes([bw])
        bases += np.uint64(base).tobytes()
        packed += oracle.ffor(d, bw, np.uint64(base)).tobytes()
    n = len(ep)
    meta = 8 + 16 + 16 * (n - 1)
    off = np.cumsum([meta, len(lanes), len(bws), len(bases)]).astype(np.uint32)
    head = bytes([5, 1, 0, 0]) + np.uint16(n).tobytes() + b"\0\0" + off.tobytes()
    head += np.array(ep[1:], np.uint32).tobytes()
    return np.frombuffer(head + lanes + bws + bases + packed + bytes(256), np.uint8)


def _constants(v):
    edge = [int(v[i]) + d for i in (0, 31, 32, 63, 64, 1023, 1024, 2047) for d in (-1, 0, 1)]
    lo, hi = (np.iinfo(v.dtype).min, np.iinfo(v.dtype).max)
    return sorted({c for c in edge + [lo, lo + 1, hi - 1, hi] if lo <= c <= hi})


@pytest.mark.parametrize("start", STARTS)
@pytest.mark.parametrize("max_gap", [0, 1, 100, 2**25])
@pytest.mark.parametrize("signed", [True, False])
def test_emulated_filter_small_deltas(start, max_gap, signed):
    emu = ctypes.CDLL(build.build())
    u = _values(start, max_gap)
    page, v = _delta_page(u), u.view(np.int64) if signed else u
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    for c in _constants(v)[::3]:
        for op in range(6):
            out = np.zeros(32, np.uint64)
            st = emu.emu_filter_page(ptr(page), ctypes.c_uint64(page.size - 256), None, ctypes.c_uint64(0), 64, 1,
                                     2 if signed else 1, ctypes.c_uint32(op), ctypes.c_uint64(c % 2**64), ptr(out))
            assert st == 0
            assert np.array_equal(out.reshape(2, 16), PR.bitmaps(v, op, c)), (c, op)


@pytest.mark.gpu
@pytest.mark.parametrize("start", STARTS)
@pytest.mark.parametrize("signed", [True, False])
def test_filter_small_deltas(cuda, start, signed):
    import torch

    from fastlanes_b200 import pages

    u = _values(start, 100)
    v, code = (u.view(np.int64), pages.INT64) if signed else (u, pages.UINT64)
    buf = torch.from_numpy(_delta_page(u).copy()).to(cuda)
    out = torch.empty(32, dtype=torch.int64, device=cuda)
    for c in _constants(v):
        for op in range(6):
            plan = pages.FilterPlan([dict(d_page=buf.data_ptr(), page_size=buf.numel() - 256, data_type=code,
                                          order=1, d_out=out.data_ptr())], op, c)
            plan.decode()
            got = out.cpu().numpy().view(np.uint64).reshape(2, 16)
            plan.close()
            assert np.array_equal(got, PR.bitmaps(v, op, c)), (c, op)


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [0, 1, 3, 8])
def test_selection_lists_edges(cuda, shift):
    """Bitmaps with no, every, one and random bits: the lists, the counts, and nothing past a list's end."""
    import torch

    from fastlanes_b200 import pages

    rng = np.random.default_rng(3)
    bits = np.zeros((9, 1024), np.uint8)
    bits[1] = 1
    bits[2, 0] = bits[3, 1023] = bits[4, 31] = bits[5, 32] = 1
    bits[6], bits[7], bits[8, 512:] = rng.random(1024) < 0.02, rng.random(1024) < 0.7, 1
    bm = torch.from_numpy(np.packbits(bits, axis=1, bitorder="little").reshape(-1)).to(cuda)
    idx = torch.full((9 * 1024 + 16,), 0x7777, dtype=torch.int16, device=cuda)
    count = torch.zeros(9, dtype=torch.int16, device=cuda)
    pages.bitmap_to_selection(bm.data_ptr(), 9, idx.data_ptr() + 2 * shift, count.data_ptr())
    want = np.full(9 * 1024 + 16, 0x7777, np.int16)
    for r in range(9):
        at = np.flatnonzero(bits[r])
        want[shift + 1024 * r:shift + 1024 * r + at.size] = at
    assert np.array_equal(idx.cpu().numpy(), want)
    assert np.array_equal(count.cpu().numpy(), bits.sum(1).astype(np.int16))
