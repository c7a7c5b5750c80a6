"""The per-row pass of string selection at its edges: symbol tables of one, two and longer symbols, shared pairs,
symbols with zero bytes and all 255 codes; empty, one-byte and long rows, rows at the column's very end, repeated
rows, and columns of different tables side by side.  The FSST page size the wizard gives holds every row's greedy
compressed length, restated here by longest match."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _table(symbols):
    """fsst_export's format of a table of these symbols (no zero-terminated mode): ordered 2..8 bytes, then 1."""
    by = [[s for s in symbols if len(s) == n] for n in (2, 3, 4, 5, 6, 7, 8, 1)]
    hist = [len(by[7])] + [len(b) for b in by[:7]]
    head = np.uint64(20190218 << 32).tobytes() + b"\0" + bytes(hist)
    return np.frombuffer(head + b"".join(b"".join(b) for b in by), np.uint8)


def _compressed(row, symbols):
    cost = p = 0
    while p < len(row):
        step = max((len(s) for s in symbols if row.startswith(s, p)), default=0)
        cost, p = (cost + 1, p + step) if step else (cost + 2, p + 1)
    return cost


TABLES = {
    "ones": [bytes([c]) for c in b"abcdef"],
    "twos": [b"ab", b"bc", b"a", b"\0\0", b"cd"],
    "long": [b"abc", b"abcd", b"abcdefgh", b"ab", b"b", b"bcd", b"abx\0", b"\0\0\0", b"h"],
    "pairs": [bytes([97 + i // 24, 97 + i % 24, 120]) for i in range(255)],
    "none": [],
}


@pytest.mark.parametrize("n_vec", [1, 5])
def test_string_rows_edges(cuda, n_vec):
    import torch

    from fastlanes_b200 import primitives as P
    from fastlanes_b200 import select as SL

    rng = np.random.default_rng(n_vec)
    cols, rows_of = [], []
    for name, symbols in TABLES.items():
        alphabet = np.frombuffer(b"abcdefghx\0\xff" if name != "pairs" else b"abcdefghijklmnopqrstuvwx", np.uint8)
        rows = [bytes(rng.choice(alphabet, int(n))) for n in rng.integers(0, 30, 1024 * n_vec)]
        for i in range(0, len(rows), 7):
            rows[i] = rows[(i * 31) % len(rows)]
        rows[3], rows[5], rows[9] = b"", b"a", bytes(rng.choice(alphabet, 5000))
        rows[-1] = b"abcdefgh"[: 1 + n_vec]
        rows_of.append((rows, symbols))
        offs = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
        data = torch.from_numpy(np.frombuffer(b"".join(rows), np.uint8).copy()).to(cuda)
        cols.append((data, torch.from_numpy(offs).to(cuda), _table(symbols)))
    plan = SL.StrSelectionPlan(cols)
    sizes = plan.wizard()[0].cpu().numpy()
    for c, (rows, symbols) in enumerate(rows_of):
        memo = {r: _compressed(r, symbols) for r in set(rows)}
        frame = 8 + 4 * 2 + 4 * 2 * (n_vec - 1)
        want = frame + sum(memo[r] for r in rows) + 4096 * n_vec + 8 + cols[c][2].size
        assert int(sizes[c, 2]) == want, list(TABLES)[c]
        assert int(sizes[c, 0]) == frame + sum(map(len, rows)) + 4096 * n_vec
    assert P.device_status() == 0
    plan.close()


@pytest.mark.parametrize("n_cols", [40, 300])
def test_string_rows_many_columns(cuda, n_cols):
    """Columns of the same strings under different tables, more vectors than the launch that fills the memo takes, and
    (300 columns) the smallest part of the memo for each."""
    import torch

    from fastlanes_b200 import primitives as P
    from fastlanes_b200 import select as SL

    rng = np.random.default_rng(n_cols)
    names = [n for n in TABLES if n != "pairs"]
    pool = [bytes(rng.choice(np.frombuffer(b"abcdefghx\0\xff", np.uint8), int(n))) for n in rng.integers(0, 30, 200)]
    cost = {name: np.array([_compressed(r, TABLES[name]) for r in pool]) for name in names}
    lens = np.array([len(r) for r in pool])
    n_vec = -(-600 // n_cols)
    cols, want, keep = [], [], {name: _table(TABLES[name]) for name in names}
    for c in range(n_cols):
        pick = rng.integers(0, len(pool), 1024 * n_vec)
        offs = np.concatenate([[0], np.cumsum(lens[pick])]).astype(np.int64)
        data = torch.from_numpy(np.frombuffer(b"".join(pool[i] for i in pick), np.uint8).copy()).to(cuda)
        name = names[c % len(names)]
        cols.append((data, torch.from_numpy(offs).to(cuda), keep[name]))
        frame = 8 + 4 * 2 + 4 * 2 * (n_vec - 1)
        want.append(frame + int(cost[name][pick].sum()) + 4096 * n_vec + 8 + keep[name].size)
    plan = SL.StrSelectionPlan(cols)
    sizes = plan.wizard()[0].cpu().numpy()
    assert [int(x) for x in sizes[:, 2]] == want
    assert P.device_status() == 0
    plan.close()
