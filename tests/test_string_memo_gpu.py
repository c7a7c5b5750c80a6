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


def _plan_of(cuda, n_cols, n_vec, rng):
    import torch

    from fastlanes_b200 import select as SL

    symbols = TABLES["long"]
    rows = [bytes(rng.choice(np.frombuffer(b"abcdefghx", np.uint8), int(n))) for n in rng.integers(0, 30, n_vec * 1024)]
    offs = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    data = torch.from_numpy(np.frombuffer(b"".join(rows), np.uint8).copy()).to(cuda)
    return SL.StrSelectionPlan([(data, torch.from_numpy(offs).to(cuda), _table(symbols))] * n_cols), rows, symbols


def _launches(call):
    import torch

    from fastlanes_b200._lib import lib

    lib.fls_gpu_launch_count(1)
    call()
    torch.cuda.synchronize()
    return lib.fls_gpu_launch_count(0)


def test_statistics_take_every_fourth_row(cuda):
    """The compressed share of a vector (statistic 1) is that of its rows 0, 4, 8, ..., in one launch over the rows."""
    plan, rows, symbols = _plan_of(cuda, 1, 200, np.random.default_rng(2))
    feat = plan.features(3)[0].cpu().numpy()
    assert _launches(lambda: plan.features(3)) == 3  # rows, integer statistics, string statistics
    for i, v in enumerate(v for c in range(0, 200, 64) for v in range(c, min(c + 64, 200), 3)):
        part = rows[v * 1024:(v + 1) * 1024]
        want = 4.0 * sum(_compressed(r, symbols) for r in part[::4]) / sum(map(len, part))
        assert abs(feat[i, 1] - want) < 1e-6 * want  # whole numbers below 2^24 in float32, one division
    plan.close()


@pytest.mark.parametrize("n_cols,n_vec,launches", [(1, 100, 1), (1, 400, 2), (18, 90, 2), (40, 30, 1), (40, 33, 2)])
def test_first_launch_only_where_it_pays(cuda, n_cols, n_vec, launches):
    """The launch that fills the memo runs for columns of 32 vectors and more, and not for so few vectors that one launch over
    all of them is all there is (on 148 SMs)."""
    import torch

    if torch.cuda.get_device_properties(cuda).multi_processor_count != 148:
        pytest.skip("the limits are those of 148 SMs")
    plan, _, _ = _plan_of(cuda, n_cols, n_vec, np.random.default_rng(3))
    assert _launches(plan.wizard) == launches + 3  # parts, dictionaries, sizes
    plan.close()
