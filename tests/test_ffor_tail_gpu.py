"""P.ffor with more widths than vectors: the bytes of the widths without a vector are zero."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_vec,n_widths", [(1, 3), (2, 3), (0, 2), (3, 3)])
def test_ffor_widths_without_vectors(cuda, n_vec, n_widths):
    import torch

    from fastlanes_b200 import primitives as P

    bw = np.array([7, 12, 31], np.uint8)[:n_widths]
    x = np.random.default_rng(3).integers(0, 128, n_vec * 1024).astype(np.uint32)
    want = np.zeros(int(bw.astype(int).sum()) * 128, np.uint8)
    at = 0
    for v in range(n_vec):
        packed = oracle.ffor(x[v * 1024:(v + 1) * 1024].copy(), int(bw[v]), np.uint32(0)).view(np.uint8)
        want[at:at + packed.size] = packed
        at += packed.size
    # the allocator hands out again what was written here
    for size in (want.size, max(want.size, 16)):
        dirty = torch.full((size,), 0xFF, dtype=torch.uint8, device=cuda)
        del dirty
    got, _ = P.ffor(torch.from_numpy(x).to(cuda), torch.from_numpy(bw).to(cuda))
    assert np.array_equal(got.cpu().numpy(), want)
