"""DICT string rows of every length the single-pass decode copies (0 to 255 bytes, dictionaries in shared and in global
memory): every offset and byte, for columns that start at every alignment of the output window and sets of columns of
very different sizes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _column(rng, n_dict, longest, n_vec, entries=None):
    lens = rng.integers(0, longest + 1, n_dict) if entries is None else np.asarray(entries)
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    data = rng.integers(0, 256, int(offs[-1]), dtype=np.uint8)
    return data, offs, rng.integers(0, lens.size, n_vec * 1024).astype(np.uint32)


def _plan(cuda, column):
    import torch

    from fastlanes_b200 import strings as S

    page, dic = S.encode_string_dict(*column)
    buf, d_dict = torch.from_numpy(page).to(cuda), torch.from_numpy(dic).to(cuda)
    return S.StringPlan(buf.data_ptr(), page.size, d_dict.data_ptr(), dic.size), (buf, d_dict)


@pytest.mark.parametrize("longest,n_dict,n_vec", [(0, 3, 1), (1, 5, 2), (9, 64, 3), (40, 4096, 5), (41, 300, 40),
                                                  (255, 256, 4), (255, 6000, 3), (100, 1, 1)])
def test_dict_rows_of_every_length(cuda, longest, n_dict, n_vec):
    from fastlanes_b200 import primitives as P
    from fastlanes_b200 import workloads as W

    rng = np.random.default_rng(longest + n_dict)
    column = _column(rng, n_dict, longest, n_vec, range(256) if (longest, n_dict) == (255, 256) else None)
    plan, keep = _plan(cuda, column)
    offs, data = plan.decode()
    assert W.dict_rows_match(offs, data, *column)
    assert P.device_status() == 0
    plan.close()


def test_set_of_uneven_columns(cuda):
    """One launch over columns of 1 to 300 vectors with dictionaries of 2 to 4,096 entries."""
    import torch

    from fastlanes_b200 import primitives as P
    from fastlanes_b200 import strings as S
    from fastlanes_b200 import workloads as W

    rng = np.random.default_rng(9)
    columns = [_column(rng, d, l, v) for d, l, v in ((2, 5, 1), (4096, 40, 300), (17, 200, 2), (1000, 12, 64), (3, 0, 5))]
    made = [_plan(cuda, c) for c in columns]
    sizes = [int(np.diff(c[1].astype(np.int64))[c[2]].sum()) for c in columns]
    offs = [torch.empty(c[2].size + 1, dtype=torch.int32, device=cuda) for c in columns]
    data = [torch.empty(n + 16, dtype=torch.uint8, device=cuda) for n in sizes]
    group = S.StringSet([p for p, _ in made])
    group.bind(offs, data)
    for _ in range(3):
        for o, d in zip(offs, data):
            o.zero_(), d.zero_()
        group.decode()
        assert all(W.dict_rows_match(o, d[:n], *c) for o, d, n, c in zip(offs, data, sizes, columns))
    assert P.device_status() == 0
    group.close()
