"""RLE, DICT and DICT_RLE pages whose indices are looked up on the way out: one to a few vectors (fewer than warps),
both orders, pages and dictionaries at every alignment (run values, codes and entries then lie off their element
size), every type the pages have."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("expr", ["rle", "dict", "dict_rle"])
@pytest.mark.parametrize("dtype", ["INT32", "UINT64"])
@pytest.mark.parametrize("n_vec", [1, 5, 200])
def test_gather_alignments(cuda, expr, dtype, n_vec):
    import torch

    from fastlanes_b200 import pages as PG
    from fastlanes_b200 import primitives as P

    code = getattr(PG, dtype)
    dt = np.dtype(PG.DTYPE_OF[code])
    rng = np.random.default_rng(n_vec)
    values = rng.integers(0, 2**31 - 1, 700, dtype=np.int64).astype(dt)
    x = np.repeat(rng.choice(values, n_vec * 1024), 1 if expr == "dict" else rng.integers(1, 9, n_vec * 1024))[:n_vec * 1024]
    x = np.ascontiguousarray(x)
    page, dic = (PG.encode_from_memory(x, code, 6)[0], None) if expr == "rle" else PG.encode_int_dict(x, expr == "dict_rle")
    ut = {4: np.uint32, 8: np.uint64}[dt.itemsize]
    tr = np.concatenate([oracle.transpose_i(x.view(ut)[v * 1024:(v + 1) * 1024].copy()) for v in range(n_vec)]).view(dt)
    for shift in range(0, 16, 3):
        buf = torch.zeros(page.size + 96, dtype=torch.uint8, device=cuda)
        buf[32 + shift:32 + shift + page.size] = torch.from_numpy(page).to(cuda)
        dbuf = None
        if dic is not None:
            dbuf = torch.zeros(dic.size + 32, dtype=torch.uint8, device=cuda)
            dbuf[shift:shift + dic.size] = torch.from_numpy(dic).to(cuda)
        for order, want in ((0, tr), (1, x)):
            out = torch.full((x.size,), -1, dtype=torch.int32 if dt.itemsize == 4 else torch.int64, device=cuda)
            PG.decode_pages([dict(d_page=buf.data_ptr() + 32 + shift, page_size=page.size, data_type=code, order=order,
                                  d_dict=None if dic is None else dbuf.data_ptr() + shift,
                                  dict_size=0 if dic is None else dic.size, d_out=out.data_ptr())])
            assert np.array_equal(out.cpu().numpy().view(dt), want), (shift, order)
    assert P.device_status() == 0
