"""FSST columns with escapes of every kind on the GPU: alone (any byte but 255 escaped), next to each other, escaped
255s, at row ends (a lone 255 decodes to a zero byte), across the 128-byte steps of the decoder, in dense and sparse
vectors side by side, at every alignment of the page; row by row against the oracle's decoder."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def _rows(rng, kind, n):
    """n compressed rows."""
    rows = []
    for _ in range(n):
        r = bytearray()
        for _ in range(int(rng.integers(0, 24))):
            x = rng.random()
            if kind == "alone" and x < 0.05:
                r += bytes([255, int(rng.integers(0, 255))])
                r.append(int(rng.integers(0, 255)))
            elif kind == "dense" and x < 0.5:
                r += bytes([255, int(rng.integers(0, 256))])
            else:
                r.append(int(rng.integers(0, 255)))
        if kind == "row_ends" and rng.random() < 0.1:
            r.append(255)
        rows.append(bytes(r))
    return rows


@pytest.mark.parametrize("shift", [0, 1, 3])
def test_fsst_escapes(cuda, col_golden, shift):
    import torch

    from fastlanes_b200 import primitives as P
    from fastlanes_b200 import strings as S

    dic = np.ascontiguousarray(col_golden["str_13_dict"])
    _, sym, ln = oracle.fsst_decode_table(dic[8:])
    rng = np.random.default_rng(shift)
    kinds = ["none", "alone", "dense", "row_ends", "alone", "none"]
    rows = [r for k in kinds for r in _rows(rng, k, 1024)]
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
