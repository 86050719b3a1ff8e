"""Rows of A on either side of the length from which a CTA slices one instead of
a warp (1100 k), alone and together; small integers, so every mode's result is
exact (8 * 8 * K < 2^24)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["split_tiled", "bf16_tiled", "tf32_tc"])
def test_rows_around_the_line(mode):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from trim_gb300 import uni10 as tu

    tu.set_stream(torch.cuda.current_stream().cuda_stream)
    rng = np.random.default_rng(17)
    shapes = [(m, 20, k) for k in (1023, 1025, 1099, 1100, 1101, 1117, 1500, 1999) for m in (1, 9, 131)]
    for group in [shapes] + [[s] for s in shapes]:
        gemms, ab, ao, bo, co = [], [], 0, 0, 0
        for m, n, k in group:
            ab.append((rng.integers(-8, 9, (m, k)).astype(np.float64), rng.integers(-8, 9, (k, n)).astype(np.float64)))
            gemms.append((m, n, k, ao, bo, co))
            ao, bo, co = ao + m * k, bo + k * n, co + m * n
        A = torch.from_numpy(np.concatenate([a.ravel() for a, _ in ab])).cuda()
        B = torch.from_numpy(np.concatenate([b.ravel() for _, b in ab])).cuda()
        C = torch.full((co,), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        tu.contract_sectors(mode, gemms, A.data_ptr(), B.data_ptr(), C.data_ptr())
        tu.sync()
        c = C.cpu().numpy()
        for (m, n, k, _, _, off), (a, b) in zip(gemms, ab):
            assert np.array_equal(c[off:off + m * n].reshape(m, n), a @ b), (m, n, k)
