"""Sets of few and of many DICT string columns, up to more than there are SMs, decoded by one launch."""
import numpy as np
import pytest

from tests.test_dict_rows_gpu import _plan

pytestmark = pytest.mark.gpu


def _column(rng, lens, n_vec):
    lens = np.asarray(lens)
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    return rng.integers(0, 256, int(offs[-1]), dtype=np.uint8), offs, rng.integers(0, lens.size, n_vec * 1024).astype(np.uint32)


@pytest.mark.parametrize("n_cols,vecs", [(2, [1, 1]), (40, [3]), (147, [5, 1]), (148, [2]), (149, [1, 9]), (600, [1, 2, 3, 40])])
def test_sets_of_columns(cuda, n_cols, vecs):
    """The same few columns many times over, decoded by one launch, several times."""
    import torch

    from fastlanes_b200 import primitives as P
    from fastlanes_b200 import strings as S
    from fastlanes_b200 import workloads as W

    rng = np.random.default_rng(n_cols)
    columns = [_column(rng, rng.integers(0, 30 + 20 * i, 20 + 300 * i), v) for i, v in enumerate(vecs)]
    made = [_plan(cuda, columns[i % len(columns)]) for i in range(n_cols)]
    sizes = [int(np.diff(c[1].astype(np.int64))[c[2]].sum()) for c in columns]
    offs = [torch.empty(columns[i % len(columns)][2].size + 1, dtype=torch.int32, device=cuda) for i in range(n_cols)]
    data = [torch.empty(sizes[i % len(columns)] + 16, dtype=torch.uint8, device=cuda) for i in range(n_cols)]
    group = S.StringSet([p for p, _ in made])
    group.bind(offs, data)
    for _ in range(2):
        for o, d in zip(offs, data):
            o.zero_(), d.zero_()
        group.decode()
        for i in range(n_cols):
            c = i % len(columns)
            if i < 2 * len(columns) or i + len(columns) >= n_cols:
                assert W.dict_rows_match(offs[i], data[i][:sizes[c]], *columns[c]), i
            else:  # equal to the first of its kind
                assert torch.equal(offs[i], offs[c]) and torch.equal(data[i][:sizes[c]], data[c][:sizes[c]]), i
    assert P.device_status() == 0
    group.close()
