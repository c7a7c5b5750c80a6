"""DICT string columns in every layout of the single-pass decode: entries padded and packed in shared memory and padded in
global memory, both windows, batches of rows that take several windows, 16- and 32-bit rows."""
import numpy as np
import pytest

from tests.test_dict_rows_gpu import _plan

pytestmark = pytest.mark.gpu


def _column(rng, lens, n_vec):
    lens = np.asarray(lens)
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    return rng.integers(0, 256, int(offs[-1]), dtype=np.uint8), offs, rng.integers(0, lens.size, n_vec * 1024).astype(np.uint32)


LENS = {
    "packed short": lambda r: np.full(200, 1),
    "packed 10000x9": lambda r: np.full(10000, 9),
    "packed 18000x5": lambda r: r.integers(4, 7, 18000),
    "global 7500": lambda r: r.integers(5, 41, 7500),
    "global 40000x9": lambda r: r.integers(8, 11, 40000),
    "padded wide 50": lambda r: r.integers(40, 61, 300),
    "padded wide 64": lambda r: r.integers(60, 69, 500),
    "padded 255": lambda r: np.full(256, 255),
    "mostly empty": lambda r: np.where(r.random(1000) < 0.9, 0, 255),
    "47 and 48": lambda r: r.integers(47, 49, 64),
    "63 and 64": lambda r: r.integers(63, 65, 64),
    "32-bit rows": lambda r: r.integers(0, 4, 70000),
    "32-bit rows, long": lambda r: r.integers(30, 90, 66000),
}


@pytest.mark.parametrize("n_vec", [1, 37])
@pytest.mark.parametrize("kind", LENS)
def test_layouts(cuda, kind, n_vec):
    from fastlanes_b200 import primitives as P
    from fastlanes_b200 import workloads as W

    rng = np.random.default_rng(len(kind) + n_vec)
    column = _column(rng, LENS[kind](rng), n_vec)
    plan, keep = _plan(cuda, column)
    offs, data = plan.decode()
    assert W.dict_rows_match(offs, data, *column)
    assert P.device_status() == 0
    plan.close()
