"""What the wizard costs by the size of its chunks: small ones have all warps too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _wizard_ms(cuda, values, chunk):
    import torch

    from fastlanes_b200 import select as SL

    plan = SL.SelectionPlan([(values, False)] * 4, chunk)
    times = []
    for _ in range(9):
        a, b = torch.cuda.Event(True), torch.cuda.Event(True)
        a.record()
        plan.wizard()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b))
    plan.close()
    return float(np.median(times[2:]))


def test_chunks_of_one_vector(cuda):
    """The same 4,096 vectors in chunks of one and of 64: 6.8 times as long with one warp a vector, twice now; one of three
    tries has to lie below the middle."""
    import torch

    v = np.minimum(np.random.default_rng(0).zipf(1.3, 1 << 20), 10**6).astype(np.int32)
    values = torch.from_numpy(v).to(cuda)
    assert any(_wizard_ms(cuda, values, 1) < 4 * _wizard_ms(cuda, values, 64) for _ in range(3))
