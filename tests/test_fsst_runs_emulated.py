"""The single-pass decode of FSST vectors with runs of escapes (fsst_total and stream_vector as k_stream_single calls them)
on an emulated warp: runs of 1 to 200 bytes 255 at every alignment and place in the decoder's 128-byte steps."""
import ctypes

import numpy as np
import pytest

from oracle import oracle
from tests import fsst_runs as R
from tests.emu import build


@pytest.fixture(scope="module")
def emu():
    return ctypes.CDLL(build.build())


@pytest.mark.parametrize("kind", ["runs", "short", "cut"])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_runs_of_escapes(emu, col_golden, kind, shift):
    _, sym, ln = oracle.fsst_decode_table(col_golden["str_13_dict"][8:])
    rng = np.random.default_rng(shift)
    rows = R.rows(rng, kind)
    comp = np.frombuffer(b"".join(rows), np.uint8)
    ends = np.cumsum([len(r) for r in rows]).astype(np.uint32)
    want = [bytes(oracle.fsst_decode(sym, ln, np.frombuffer(r, np.uint8))) for r in rows]
    buf = np.full(comp.size + 32, 0xFF, np.uint8)
    at = (-buf.ctypes.data) % 16 + shift
    buf[at:at + comp.size] = comp
    vbase = 5 + shift
    out = np.full(vbase + sum(map(len, want)) + 64, 0xEE, np.uint8)
    offs = np.zeros(1025, np.uint32)
    got, lone = ctypes.c_uint64(), ctypes.c_int()
    P = lambda a: ctypes.c_void_p(a.ctypes.data)
    emu.emu_stream_single.restype = ctypes.c_uint64
    # window stores go to 16-byte aligned output
    raw = np.full(out.size + 16, 0xEE, np.uint8)
    o = (-raw.ctypes.data) % 16
    total = emu.emu_stream_single(P(np.ascontiguousarray(sym)), P(np.ascontiguousarray(ln)), P(ends),
                                  ctypes.c_void_p(buf.ctypes.data + at), ctypes.c_uint32(comp.size), ctypes.c_uint64(vbase),
                                  P(offs), ctypes.c_void_p(raw.ctypes.data + o), ctypes.byref(got), ctypes.byref(lone))
    n = sum(map(len, want))
    assert total == got.value == n
    assert (lone.value == 1) == (kind == "short")  # runs of 64 and more, and cut ones, take the general walk
    assert raw[o + vbase:o + vbase + n].tobytes() == b"".join(want)
    assert (raw[o:o + vbase] == 0xEE).all() and (raw[o + vbase + n:] == 0xEE).all()
    assert offs.tolist() == (vbase + np.concatenate([[0], np.cumsum([len(w) for w in want])])).tolist()
