"""FSST columns with runs of 1 to 200 escapes on the GPU, whole and cut by row ends, at every alignment of the page."""
import numpy as np
import pytest

from oracle import oracle
from tests import fsst_runs as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_runs_of_escapes(cuda, col_golden, shift):
    import torch

    from fastlanes_b200 import primitives as P
    from fastlanes_b200 import strings as S

    dic = np.ascontiguousarray(col_golden["str_13_dict"])
    _, sym, ln = oracle.fsst_decode_table(dic[8:])
    rng = np.random.default_rng(10 + shift)
    rows = [r for kind in ("runs", "short", "cut", "short") for r in R.rows(rng, kind)]
    coffs = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint64)
    page, _ = S.fsst_page(dic[8:], np.frombuffer(b"".join(rows), np.uint8), coffs)
    want = [bytes(oracle.fsst_decode(sym, ln, np.frombuffer(r, np.uint8))) for r in rows]
    buf = torch.zeros(page.size + 32, dtype=torch.uint8, device=cuda)
    buf[shift:shift + page.size] = torch.from_numpy(page).to(cuda)
    d_dict = torch.from_numpy(dic).to(cuda)
    plan = S.StringPlan(buf.data_ptr() + shift, page.size, d_dict.data_ptr(), dic.size)
    offs, data = plan.decode()
    assert offs.tolist() == np.concatenate([[0], np.cumsum([len(w) for w in want])]).tolist()
    assert data.cpu().numpy().tobytes() == b"".join(want)
    assert P.device_status() == 0
    plan.close()
