"""Maxima and digit images of the tensor-core modes over every path of the
one-pass slicing: rows a warp stages (K <= 1024), reads twice (to 2000) or a
CTA stages (to 8192), strips of 16 columns staged (K <= 576) or read twice, and
the tile-by-tile form of a few rows of long K; zero and subnormal rows and
columns.  The operands are small integers times a power of two per row and
column, so every mode's products and FP32 sums are exact (8 * 8 * K < 2^24) and
the result is the integer product, scaled, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [
    (1, 1, 1), (9, 17, 15), (8, 16, 16), (130, 66, 17), (7, 33, 575), (17, 15, 576), (5, 18, 577), (129, 65, 1023),
    (3, 40, 1024), (12, 16, 1025), (40, 31, 1999), (9, 9, 2000), (10, 20, 2001), (6, 70, 8192), (4, 3, 8193),
]


@pytest.fixture(scope="module")
def env():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from trim_gb300 import uni10 as tu

    tu.set_stream(torch.cuda.current_stream().cuda_stream)
    return torch, tu


@pytest.mark.parametrize("mode", ["split_tiled", "bf16_tiled", "tf32_tc"])
@pytest.mark.parametrize("grouped", [False, True])
def test_exact_products(env, mode, grouped):
    torch, tu = env
    rng = np.random.default_rng(41)
    for shapes in ([SHAPES * 12] if grouped else [[s] for s in SHAPES]):
        gemms, ao, bo, co, ab, want = [], 0, 0, 0, [], []
        for m, n, k in shapes:
            a = rng.integers(-8, 9, (m, k)).astype(np.float64)
            b = rng.integers(-8, 9, (k, n)).astype(np.float64)
            a[m // 2] = 0.0  # a zero row, a zero column
            b[:, n // 3] = 0.0
            ra, cb = rng.integers(-30, 30, (m, 1)), rng.integers(-30, 30, (1, n))
            ra[0] = -1060  # subnormal values: 8 * 2^-1060 and below
            want.append(np.ldexp(a @ b, ra + cb))
            ab.append((np.ldexp(a, ra), np.ldexp(b, cb)))
            gemms.append((m, n, k, ao, bo, co))
            ao, bo, co = ao + m * k, bo + k * n, co + m * n
        A = torch.from_numpy(np.concatenate([a.ravel() for a, _ in ab])).cuda()
        B = torch.from_numpy(np.concatenate([b.ravel() for _, b in ab])).cuda()
        C = torch.full((co,), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        tu.contract_sectors(mode, gemms, A.data_ptr(), B.data_ptr(), C.data_ptr())
        tu.sync()
        c = C.cpu().numpy()
        for (m, n, k, _, _, off), w in zip(gemms, want):
            assert np.array_equal(c[off:off + m * n].reshape(m, n), w), (mode, m, n, k)


@pytest.mark.parametrize("mode", ["bf16_tiled", "tf32_tc", "split_tiled"])
@pytest.mark.parametrize("m,n,k", [(9000, 323, 70), (19400, 577, 33), (2050, 1300, 129), (640, 4100, 64), (8, 9728, 8300)])
def test_wide_items_exact(env, mode, m, n, k):
    """Enough output tiles for items of two and four column tiles, the last of
    them ragged, and two K ranges of more than 4096 k; small integers, so every
    mode's result is exact."""
    torch, tu = env
    rng = np.random.default_rng(m)
    a = rng.integers(-8, 9, (m, k)).astype(np.float64)
    b = rng.integers(-8, 9, (k, n)).astype(np.float64)
    A, B = torch.from_numpy(a.ravel()).cuda(), torch.from_numpy(b.ravel()).cuda()
    C = torch.full((m * n,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    tu.contract_sectors(mode, [(m, n, k, 0, 0, 0)], A.data_ptr(), B.data_ptr(), C.data_ptr())
    tu.sync()
    assert np.array_equal(C.cpu().numpy().reshape(m, n), a @ b)
