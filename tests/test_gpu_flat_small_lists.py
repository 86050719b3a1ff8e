"""FP64 lists too small to fill the GPU: sectors of up to eight columns as rows
(one to a warp, four at a time, with K ranges), few outputs with K ranges and
their sums, and such sectors in a list of more items than the GPU holds warps,
against a numpy product.  Any order of K products and sums errs by at most
K 2^-53 of the sum of magnitudes (to first order), here and in the reference."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LISTS = [[(m, n, k)] for n in range(1, 10) for m, k in ((1, 33), (3, 64), (13, 97), (5, 700), (2, 9001))]
LISTS += [[(m, n, k) for n in range(1, 10) for m in (1, 4, 7) for k in (31, 32, 65, 500)]]
LISTS += [[(735, n, 40)] * 12 for n in (1, 2, 3, 8)] + [[(85 + i, 1 + i % 3, 60) for i in range(100)]]
LISTS += [[(16, 2, 23723)], [(5, 9, 23723)], [(4, 13, 23723)], [(3, 7, 14786)], [(9, 16, 320)] * 20]


def test_small_lists():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from trim_gb300 import uni10 as tu

    tu.set_stream(torch.cuda.current_stream().cuda_stream)
    rng = np.random.default_rng(53)
    for shapes in LISTS:
        gemms, ao, bo, co = [], 0, 0, 0
        for m, n, k in shapes:
            gemms.append((m, n, k, ao, bo, co))
            ao, bo, co = ao + m * k, bo + k * n, co + m * n
        a, b = rng.uniform(-1, 1, ao), rng.uniform(-1, 1, bo)
        A, B = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
        outs = []
        for _ in range(2):
            C = torch.full((co,), float("nan"), dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            tu.contract_sectors("fp64", gemms, A.data_ptr(), B.data_ptr(), C.data_ptr())
            tu.sync()
            outs.append(C.cpu().numpy())
        assert np.array_equal(outs[0], outs[1])
        for m, n, k, oa, ob, oc in gemms:
            x, y = a[oa:oa + m * k].reshape(m, k), b[ob:ob + k * n].reshape(k, n)
            err = np.abs(outs[0][oc:oc + m * n].reshape(m, n) - x @ y)
            assert np.all(err <= 2 * (k + 1) * 2.0 ** -53 * (np.abs(x) @ np.abs(y))), (m, n, k, len(shapes))
