"""Row statistics of string columns side by side: what a vector costs does not grow with the number of columns."""
import numpy as np
import pytest

from tests.test_string_rows_gpu import TABLES, _table

pytestmark = pytest.mark.gpu


def _features_ms(cuda, n_cols, n_vec):
    import torch

    from fastlanes_b200 import select as SL

    rng = np.random.default_rng(1)
    rows = n_vec * 1024
    offs = torch.from_numpy(np.arange(0, 12 * rows + 1, 12)).to(cuda)
    data = torch.from_numpy(rng.integers(97, 105, 12 * rows, dtype=np.uint8)).to(cuda)
    plan = SL.StrSelectionPlan([(data, offs, _table(TABLES["long"]))] * n_cols)
    times = []
    for _ in range(7):
        a, b = torch.cuda.Event(True), torch.cuda.Event(True)
        a.record()
        plan.features(1)
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b))
    plan.close()
    return float(np.median(times[2:]))


def test_many_columns_of_one_vector(cuda):
    """1,500 columns of one vector beside one column of 1,500: a symbol table for each of them, and no more.  Measured 2 to
    3 times as long; 40 times when every CTA looked at every column."""
    assert any(_features_ms(cuda, 1500, 1) < 8 * _features_ms(cuda, 1, 1500) for _ in range(3))
