"""The flat FP64 grouped GEMM (a warp per item, outputs dealt to lanes) at its
edges: outputs around the 32-lane slot and the 128-output rule, one and two
columns (lanes along K), K around 32 and long enough for K ranges and their
partial sums, alone and grouped, against a numpy product.  Any order of K
products and sums of a dot product errs by at most K 2^-53 of the sum of
magnitudes (to first order), for the kernel and for the reference alike."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [
    (1, 1, 1), (1, 1, 31), (3, 1, 32), (65, 1, 33), (5, 2, 100), (2, 2, 31), (4, 8, 64), (1, 32, 40), (33, 1, 4097),
    (10, 10, 1), (10, 10, 1000), (11, 3, 2500), (7, 18, 129), (32, 4, 65), (127, 1, 7), (8, 16, 5000), (3, 43, 200),
    (29, 28, 2500), (130, 130, 130), (31, 33, 64), (257, 5, 17), (64, 64, 8), (100, 100, 3000),
]


@pytest.fixture(scope="module")
def env():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from trim_gb300 import uni10 as tu

    tu.set_stream(torch.cuda.current_stream().cuda_stream)
    return torch, tu


@pytest.mark.parametrize("copies", [0, 1, 40])
def test_flat_fp64_edges(env, copies):
    """copies 0: every sector by itself; 1: all in one list; 40: a list long
    enough that warps take several items, twice for the reset of the groups."""
    torch, tu = env
    rng = np.random.default_rng(23)
    batches = [[s] for s in SHAPES] if copies == 0 else [SHAPES * copies]
    for shapes in batches:
        gemms, ao, bo, co = [], 0, 0, 0
        for m, n, k in shapes:
            gemms.append((m, n, k, ao, bo, co))
            ao, bo, co = ao + m * k, bo + k * n, co + m * n
        a, b = rng.uniform(-1, 1, ao), rng.uniform(-1, 1, bo)
        A, B = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
        C = torch.full((co,), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        outs = []
        for _ in range(2):
            tu.contract_sectors("fp64", gemms, A.data_ptr(), B.data_ptr(), C.data_ptr())
            tu.sync()
            outs.append(C.cpu().numpy())
        assert np.array_equal(outs[0], outs[1])
        for m, n, k, oa, ob, oc in gemms:
            x, y = a[oa:oa + m * k].reshape(m, k), b[ob:ob + k * n].reshape(k, n)
            err = np.abs(outs[0][oc:oc + m * n].reshape(m, n) - x @ y)
            assert np.all(err <= 2 * (k + 1) * 2.0 ** -53 * (np.abs(x) @ np.abs(y))), (m, n, k)
