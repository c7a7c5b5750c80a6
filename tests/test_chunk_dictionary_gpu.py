"""The wizard's chunk dictionary on the GPU at the edges of its table: chunks of one to 64 vectors whose distinct
values all fit, just fit, just do not, or arrive late, with the extreme keys of each type and keys that differ in
few bits; the distinct counts and the DICT sizes (every vector's code width) against the oracle."""
import numpy as np
import pytest

from oracle import select as OS

pytestmark = pytest.mark.gpu

KINDS = ("distinct", "constant", "late", "high_bits", "low_bits", "extremes", "repeats")


def _values(kind, n_vec, width, rng):
    n = n_vec * 1024
    ut = {32: np.uint32, 64: np.uint64}[width]
    if kind == "distinct":
        return rng.permutation(n).astype(ut) * ut(2654435761)
    if kind == "constant":
        return np.full(n, 2**width - 1, ut)
    if kind == "late":  # few values for half of the chunk, every value new after
        x = np.arange(n, dtype=ut) + ut(1000)
        x[: n // 2] = rng.integers(0, 50, n // 2)
        return x
    if kind == "high_bits":
        return rng.integers(0, 60000, n).astype(ut) << ut(width - 16)
    if kind == "low_bits":
        return rng.integers(0, 60000, n).astype(ut)
    if kind == "extremes":
        return rng.choice(np.array([0, 1, 2**(width - 1) - 1, 2**(width - 1), 2**width - 2, 2**width - 1], ut), n)
    return np.repeat(rng.integers(0, 2**width - 1, n // 4 + 1, dtype=np.uint64).astype(ut), 4)[:n]


@pytest.mark.parametrize("width", [32, 64])
@pytest.mark.parametrize("n_vec", [1, 3, 8, 9, 44, 45, 64])
def test_chunk_dictionary_edges(cuda, width, n_vec):
    import torch

    from fastlanes_b200 import primitives as P
    from fastlanes_b200 import select as SL

    rng = np.random.default_rng(width + n_vec)
    host = [_values(k, n_vec, width, rng) for k in KINDS]
    st = {32: np.int32, 64: np.int64}[width]
    plan = SL.SelectionPlan([(torch.from_numpy(v.view(st)).to(cuda), False) for v in host])
    sizes, _, distinct = plan.wizard()
    sizes, distinct = sizes.cpu().numpy(), distinct.cpu().numpy()
    for i, v in enumerate(host):
        d, codes = OS.chunk_dictionary(v)
        code_bits = sum(int(c.max() - c.min()).bit_length() for c in codes.reshape(n_vec, 1024).astype(np.int64))
        want = 20 + d * (width // 8) + 8 + 17 * n_vec + 128 * code_bits
        assert (int(distinct[i]), int(sizes[i, 4])) == (d, want), KINDS[i]
    assert P.device_status() == 0
    plan.close()


def _filter_place(lo, hi):
    """Where the filter of nearly unique chunks puts a 64-bit key (the kernel's hash, restated)."""
    with np.errstate(over="ignore"):
        a = lo * np.uint32(0x9E3779B1) + hi * np.uint32(0x85EBCA77)
        a = (a ^ (a >> np.uint32(15))) * np.uint32(0x2C1B3C6D)
        return (a ^ (a >> np.uint32(13))) >> np.uint32(12)


@pytest.mark.parametrize("kind", ["few_repeats", "many_repeats", "one_filter_bit", "shared_marks"])
def test_chunk_dictionary_nearly_unique(cuda, kind):
    """Chunks around the limits of the unique path: a few and too many repeats, every key on one filter bit, and
    unique keys crowded onto few marks so that the marked values overflow their table."""
    import torch

    from fastlanes_b200 import primitives as P
    from fastlanes_b200 import select as SL

    rng = np.random.default_rng(5)
    n = 64 * 1024
    v = rng.permutation(np.unique(rng.integers(0, 2**63, n + 100, dtype=np.uint64))[:n])
    if kind in ("few_repeats", "many_repeats"):
        k = 3000 if kind == "few_repeats" else 12000
        v[rng.integers(0, n, k)] = v[rng.integers(0, n, k)]
    else:
        lo = rng.integers(0, 2**32, 1 << 24, dtype=np.uint64).astype(np.uint32)
        place = _filter_place(lo, np.uint32(7))
        if kind == "one_filter_bit":
            some = np.unique(lo[place == 77])
        else:  # keys of one mark in eight: a key on each of its four filter bits, and one more that finds its bit set
            some = np.unique(lo[(place >> np.uint32(2)) % 32 == 0])
        v[: min(n, some.size)] = rng.permutation(some)[:n].astype(np.uint64) | np.uint64(7 << 32)
    plan = SL.SelectionPlan([(torch.from_numpy(v.view(np.int64)).to(cuda), False)])
    sizes, _, distinct = plan.wizard()
    d, codes = OS.chunk_dictionary(v)
    code_bits = sum(int(c.max() - c.min()).bit_length() for c in codes.reshape(64, 1024).astype(np.int64))
    assert (int(distinct[0]), int(sizes[0, 4])) == (d, 20 + 8 * d + 8 + 17 * 64 + 128 * code_bits)
    assert P.device_status() == 0
    plan.close()
