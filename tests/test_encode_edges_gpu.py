"""Encoder primitives at their edges: transposing one vector, odd counts and buffers that are not 16-byte aligned;
packing every bit width of every type; the packed offsets around the scan's turns and alignments."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu
TYPES = {8: np.uint8, 16: np.uint16, 32: np.uint32, 64: np.uint64}


@pytest.mark.parametrize("w", [8, 16, 32, 64])
@pytest.mark.parametrize("n,shift", [(1, 0), (3, 0), (5, 1), (9, 3)])
def test_transpose_alignments(cuda, w, n, shift):
    import torch

    from fastlanes_b200._lib import lib

    x = np.random.default_rng(w + n).integers(0, np.iinfo(TYPES[w]).max, n * 1024, dtype=np.uint64).astype(TYPES[w])
    step = w // 8
    src = torch.zeros(n * 1024 * step + 64, dtype=torch.uint8, device=cuda)
    src[shift * step:shift * step + x.nbytes] = torch.from_numpy(x.view(np.uint8)).to(cuda)
    dst = torch.full((n * 1024 * step + 64,), 0xA5, dtype=torch.uint8, device=cuda)
    rc = getattr(lib, f"fls_gpu_transpose_i_u{w}")(src.data_ptr() + shift * step, dst.data_ptr() + shift * step, n, None)
    assert rc == 0
    got = dst.cpu().numpy()
    want = np.concatenate([oracle.transpose_i(x[v * 1024:(v + 1) * 1024].copy()) for v in range(n)])
    assert np.array_equal(got[shift * step:shift * step + x.nbytes], want.view(np.uint8))
    assert (got[:shift * step] == 0xA5).all() and (got[shift * step + x.nbytes:] == 0xA5).all()


@pytest.mark.parametrize("w", [8, 16, 32, 64])
def test_ffor_every_width(cuda, w):
    import torch

    from fastlanes_b200 import primitives as P

    rng = np.random.default_rng(w)
    bw = rng.permutation(w + 1).astype(np.uint8)
    base = rng.integers(0, np.iinfo(TYPES[w]).max, w + 1, dtype=np.uint64).astype(TYPES[w])
    x = rng.integers(0, 2**64 - 1, (w + 1, 1024), dtype=np.uint64)
    x &= (np.uint64(2**64 - 1) >> (np.uint64(64) - np.maximum(bw, 1).astype(np.uint64)))[:, None]
    x[bw == 0] = 0
    vals = (x.astype(TYPES[w]) + base[:, None]).astype(TYPES[w])
    to = lambda a: torch.from_numpy(a).to(cuda)
    packed, off = P.ffor(to(vals.reshape(-1)), to(bw), to(base))
    want = [oracle.ffor(vals[v], int(bw[v]), base[v]).view(np.uint8) for v in range(w + 1)]
    assert np.array_equal(packed.cpu().numpy(), np.concatenate(want))
    assert off.view(torch.int64).tolist() == np.cumsum([0] + [a.size for a in want])[:-1].tolist()


@pytest.mark.parametrize("n", [0, 1, 15, 16, 17, 16383, 16384, 16385, 40000])
@pytest.mark.parametrize("shift", [0, 5])
def test_pack_offsets(cuda, n, shift):
    import torch

    from fastlanes_b200._lib import lib

    bw = np.random.default_rng(n).integers(0, 65, n + shift).astype(np.uint8)
    d_bw = torch.from_numpy(bw).to(cuda)
    off = torch.full((n + 1,), -7, dtype=torch.int64, device=cuda)
    for width in (64, 40):
        total = torch.full((2,), -1, dtype=torch.int64, device=cuda)
        assert lib.fls_gpu_pack_offsets(d_bw.data_ptr() + shift, n, width, off.data_ptr(), total.data_ptr(), None) == 0
        ends = np.cumsum(bw[shift:].astype(np.int64) * 128)
        assert off.tolist() == np.concatenate([[0], ends])[:n].tolist() + [-7]
        assert total.tolist() == [int(ends[-1]) if n else 0, int((bw[shift:] > width).any())]


def test_ffor_impossible_width_leaves_zeros(cuda):
    import torch

    from fastlanes_b200 import primitives as P

    x = torch.arange(2048, dtype=torch.int32, device=cuda).view(torch.uint32)
    packed, _ = P.ffor(x, torch.tensor([33, 5], dtype=torch.uint8, device=cuda))
    assert packed.numel() == 38 * 128 and not packed[:33 * 128].any()
