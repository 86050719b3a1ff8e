"""Split, BF16 and TF32 contractions of many short rows (K below about 120,
sliced in two launches) and of the same K as columns (in one), at ragged sizes;
small integers, so every mode's result is exact (8 * 8 * K < 2^24)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["split_tiled", "bf16_tiled", "tf32_tc"])
@pytest.mark.parametrize("m,n,k,copies", [(70001, 24, 41, 1), (150003, 17, 16, 1), (19, 60007, 33, 1), (9557, 24, 41, 9), (40009, 33, 127, 1),
                                          (40009, 33, 200, 1)])
def test_short_rows(mode, m, n, k, copies):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from trim_gb300 import uni10 as tu

    tu.set_stream(torch.cuda.current_stream().cuda_stream)
    g = torch.Generator(device="cuda").manual_seed(m)
    a, b = (torch.randint(-8, 9, (v,), generator=g, device="cuda").double() for v in (copies * m * k, copies * k * n))
    c = torch.full((copies * m * n,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    tu.contract_sectors(mode, [(m, n, k, i * m * k, i * k * n, i * m * n) for i in range(copies)], a.data_ptr(), b.data_ptr(), c.data_ptr())
    tu.sync()
    assert torch.equal(c.view(copies, m, n), torch.bmm(a.view(copies, m, k), b.view(copies, k, n)))
