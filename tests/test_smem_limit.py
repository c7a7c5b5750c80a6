"""A kernel's dynamic shared-memory limit is set on every device it is launched on (a fake of the runtime's calls)."""
import ctypes

import numpy as np

from tests.emu import build


def test_limit_is_set_per_device():
    emu = ctypes.CDLL(build.build())
    device = np.array([0, 0, 1, 0, 1, 63, 0, 1, 64, -1], np.int32)
    size = np.array([60000, 60000, 60000, 70000, 65000, 1, 60000, 70000, 100, 100], np.uint32)
    asked, error = np.full(10, -1, np.int32), np.full(10, -1, np.int32)
    P = lambda a: ctypes.c_void_p(a.ctypes.data)
    emu.emu_smem_limit(P(device), P(size), 10, P(asked), P(error))
    assert asked.tolist() == [60000, 0, 60000, 70000, 65000, 1, 0, 70000, 0, 0]
    assert error.tolist() == [0] * 8 + [101] * 2


def test_launchers_keep_no_flag_of_their_own():
    """Every launcher that raises the limit does it through the per-device one."""
    import pathlib

    src = pathlib.Path(__file__).parent.parent / "fastlanes_b200" / "csrc"
    for name in ("fls_k_select.cu", "fls_k_strings.cu"):
        assert "cudaFuncSetAttribute" not in (src / name).read_text(), name
