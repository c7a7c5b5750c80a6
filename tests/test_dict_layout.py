"""How the single-pass DICT decode lays out its CTAs (dict_layout), on the CPU: the shared memory holds what the kernel
puts there, and padding entries or a wider window costs no column more warps than it is worth."""
import ctypes

import numpy as np
import pytest

from tests.emu import build

GLOBAL, SMEM8, PACKED = 0, 1, 2


@pytest.fixture(scope="module")
def layout():
    emu = ctypes.CDLL(build.build())
    emu.emu_dict_layout.argtypes = [ctypes.c_uint64] * 4 + [ctypes.c_int, ctypes.c_void_p]

    def f(lens, rows16=True):
        lens = np.asarray(lens)
        out = np.zeros(6, np.uint32)
        packed = int(lens.sum())
        emu.emu_dict_layout(int(((lens + 7) // 8 * 8).sum()), packed, lens.size, packed // lens.size, int(rows16),
                            out.ctypes.data)
        return dict(zip(("mode", "warps", "window", "dict_cap", "smem", "rows"), out.tolist()))

    return f


@pytest.mark.parametrize("rows16", [True, False])
def test_shared_memory_holds_everything(layout, rows16):
    rng = np.random.default_rng(4)
    for _ in range(3000):
        n = int(2 ** rng.uniform(0, 17))
        lens = rng.integers(0, int(2 ** rng.uniform(0, 8)) + 1, n) if rng.random() < 0.8 else np.zeros(n, int)
        l = layout(lens, rows16)
        tab = (4 * n + 15) // 16 * 16
        need = l["warps"] * (l["rows"] + l["window"])
        if l["mode"] != GLOBAL:
            held = int(((lens + 7) // 8 * 8).sum() if l["mode"] == SMEM8 else lens.sum())
            assert l["dict_cap"] % 16 == 0 and l["dict_cap"] >= held and l["warps"] >= 13
            need += l["dict_cap"] + tab
        assert l["window"] % 16 == 0 and l["window"] >= 255 + 15 and 1 <= l["warps"] <= 32
        assert l["smem"] == need and need <= 226 * 1024


@pytest.mark.parametrize("entries,length,mode,window,warps", [
    (10000, 9, PACKED, 1536, 25), (18000, 5, PACKED, 1536, 18), (12000, 4, PACKED, 2048, 32), (200, 1, PACKED, 2048, 32),
    (6000, 17, PACKED, 1536, 28), (300, 25, SMEM8, 2048, 32), (4096, 22, SMEM8, 1536, 30), (300, 50, SMEM8, 2048, 32),
    (2000, 55, SMEM8, 2048, 25), (40000, 9, GLOBAL, 1536, 32), (7500, 23, GLOBAL, 1536, 32), (300, 0, PACKED, 2048, 32)])
def test_choices(layout, entries, length, mode, window, warps):
    l = layout(np.full(entries, length))
    assert (l["mode"], l["window"]) == (mode, window) and l["warps"] >= warps
