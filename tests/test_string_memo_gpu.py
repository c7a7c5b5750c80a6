"""Compressed lengths of rows that share a hash: string selection takes a row's from another row only when their bytes are
the same."""
import numpy as np
import pytest

from tests.test_string_rows_gpu import TABLES, _compressed, _table

pytestmark = pytest.mark.gpu
M64 = 2**64 - 1
SEED, STEP = 0x243F6A8885A308D3, 0x9E3779B97F4A7C15


def _mix(h):
    """The 64-bit finaliser of MurmurHash3."""
    h ^= h >> 33
    h = h * 0xFF51AFD7ED558CCD & M64
    h ^= h >> 33
    h = h * 0xC4CEB9FE1A85EC53 & M64
    return h ^ h >> 33


def _twin(row, first):
    """A row of 16 bytes with `first` in front whose hash is that of `row`, if the second word takes up the first one's
    difference as it does in a hash of xor and bijections."""
    word = lambda b: int.from_bytes(b, "little")
    h = [(_mix(SEED ^ 16 ^ word(x)) + STEP) & M64 for x in (row[:8], first)]
    return first + (word(row[8:]) ^ h[0] ^ h[1]).to_bytes(8, "little")


@pytest.mark.parametrize("n_vec", [3, 400])
def test_rows_of_one_hash(cuda, n_vec):
    import torch

    from fastlanes_b200 import primitives as P
    from fastlanes_b200 import select as SL

    symbols = TABLES["long"]
    a = b"abcdefghabcdefgh"
    rows = [a, _twin(a, b"xxxxxxxx"), b"abcd", _twin(a, b"hhhhhhhh"), b"", b"a" * 3000, b"ab" * 1023, b"ab" * 1024]
    assert len({_compressed(r, symbols) for r in rows[:2] + rows[3:4]}) > 1
    rng = np.random.default_rng(n_vec)
    pick = rng.choice(len(rows), n_vec * 1024, p=[.3, .3, .1, .2, .09, .003, .004, .003])
    lens = np.array([len(r) for r in rows])
    offs = np.concatenate([[0], np.cumsum(lens[pick])]).astype(np.int64)
    data = torch.from_numpy(np.frombuffer(b"".join(rows[i] for i in pick), np.uint8).copy()).to(cuda)
    table = _table(symbols)
    plan = SL.StrSelectionPlan([(data, torch.from_numpy(offs).to(cuda), table)])
    cost = np.array([_compressed(r, symbols) for r in rows])
    sizes = plan.wizard()[0].cpu().numpy().reshape(-1, 6)
    for c in range(sizes.shape[0]):
        part = pick[c * 65536:(c + 1) * 65536]
        nv = part.size // 1024
        frame = 8 + 4 * 2 + 4 * 2 * (nv - 1)
        assert int(sizes[c, 2]) == frame + int(cost[part].sum()) + 4096 * nv + 8 + table.size
        assert int(sizes[c, 0]) == frame + int(lens[part].sum()) + 4096 * nv
    assert P.device_status() == 0
    plan.close()
