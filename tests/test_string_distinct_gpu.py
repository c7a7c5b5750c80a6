"""Distinct rows of a string chunk: short rows whose length cancels against their bytes in the rows' hash ("a" and "b"
with a zero byte), in DICT sizes, distinct counts and runs."""
import numpy as np
import pytest

from tests.test_string_rows_gpu import _compressed, _table

pytestmark = pytest.mark.gpu


def _pairs():
    """Rows of 1 to 12 bytes, and longer ones of the same bytes with zeros behind, the first byte changed by the xor of the
    two lengths."""
    out = []
    for row in (b"a", b"gg", b"abc", b"abcdefg", b"abcdefgh", b"abcdefghi", b"abcdefghijkl", b"q\0"):
        out.append(row)
        for m in range(len(row) + 1, -(-len(row) // 8) * 8 + 1):
            out.append(bytes([row[0] ^ len(row) ^ m]) + row[1:] + b"\0" * (m - len(row)))
    return sorted(set(out))


@pytest.mark.parametrize("n_vec", [1, 3])
def test_rows_that_end_in_zero_bytes(cuda, n_vec):
    import torch

    from fastlanes_b200 import primitives as P
    from fastlanes_b200 import select as SL

    rng = np.random.default_rng(n_vec)
    pool = _pairs()
    symbols = [b"abc", b"gh", b"\0\0", b"a"]
    pick = rng.integers(0, len(pool), n_vec * 1024)
    rows = [pool[i] for i in pick]
    offs = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    data = torch.from_numpy(np.frombuffer(b"".join(rows), np.uint8).copy()).to(cuda)
    plan = SL.StrSelectionPlan([(data, torch.from_numpy(offs).to(cuda), _table(symbols))])
    sizes, _, distinct = plan.wizard()
    sizes, distinct = sizes.cpu().numpy()[0], int(distinct[0])
    code = {}
    for r in rows:
        code.setdefault(r, len(code))
    codes = np.array([code[r] for r in rows]).reshape(n_vec, 1024)
    code_bits = sum(int(c.max() - c.min()).bit_length() for c in codes)
    runs = sum(1 + int((c[1:] != c[:-1]).sum()) for c in codes)
    frame = lambda arr: 8 + 4 * arr + 4 * arr * (n_vec - 1)
    dic = 8 + 2066 + 4 * len(code) + sum(_compressed(r, symbols) for r in code)
    assert distinct == len(code)
    assert int(sizes[1]) == frame(3) + n_vec + 4 * n_vec + 128 * code_bits + dic
    assert int(sizes[3]) == frame(2) + 4 * runs + 2048 * n_vec + dic
    assert P.device_status() == 0
    plan.close()
