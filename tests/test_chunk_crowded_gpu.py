"""Chunks whose keys crowd in the wizard's table, by structure or chosen against its hash: exact all the same."""
import numpy as np
import pytest

from oracle import select as OS
from tests import chunk_keys as CK

pytestmark = pytest.mark.gpu


def _halves(n, rng):
    i = rng.permutation(n).astype(np.uint64)
    return ((i >> np.uint64(8)) << np.uint64(56)) | ((i & np.uint64(255)) << np.uint64(24))


def _deep_repeats(n, rng):
    """Rows of 20 new keys and 12 of the first ones, all on one place."""
    k = CK.key64(9, np.arange(n))
    x = k.copy().reshape(-1, 32)
    few = min(n, 4000)
    x[:, 20:] = k[:few][rng.integers(0, few, (n // 32, 12))]
    return x.reshape(-1)


KEYS = {
    "halves": _halves,
    "one_place_64": lambda n, rng: rng.permutation(CK.key64(77, np.arange(n))),
    "one_part_64": lambda n, rng: rng.permutation(CK.key64(rng.integers(0, 2**32, n, dtype=np.uint64), np.arange(n))),
    "one_place_32": lambda n, rng: rng.permutation(CK.key32(np.arange(n))),
    "one_part_32": lambda n, rng: rng.permutation(CK.key32(np.arange(n) * 65536)),
    "deep_repeats": _deep_repeats,
    "two_values": lambda n, rng: np.where(np.arange(n) % 32 == 7, CK.key64(3, 1), CK.key64(3, 2)),
}


@pytest.mark.parametrize("n_vec", [1, 3, 21, 64])
@pytest.mark.parametrize("kind", KEYS)
def test_crowded_keys(cuda, kind, n_vec):
    import torch

    from fastlanes_b200 import primitives as P
    from fastlanes_b200 import select as SL

    n = n_vec * 1024
    v = np.ascontiguousarray(KEYS[kind](n, np.random.default_rng(n)))
    width = v.itemsize
    plan = SL.SelectionPlan([(torch.from_numpy(v.view({4: np.int32, 8: np.int64}[width])).to(cuda), False)])
    sizes, _, distinct = plan.wizard()
    d, codes = OS.chunk_dictionary(v)
    code_bits = sum(int(c.max() - c.min()).bit_length() for c in codes.reshape(n_vec, 1024).astype(np.int64))
    assert (int(distinct[0]), int(sizes[0, 4])) == (d, 20 + d * width + 8 + 17 * n_vec + 128 * code_bits)
    assert P.device_status() == 0
    plan.close()
