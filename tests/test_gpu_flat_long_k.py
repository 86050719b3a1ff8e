"""FP64 sectors of one, two or a few outputs over a long K (a norm, an
expectation value, the last contraction of a network): K ranges on many warps
and their sums, alone and beside others, twice for the reset of the groups,
against a numpy product.  Any order of K products and sums errs by at most
K 2^-53 of the sum of magnitudes (to first order), here and in the reference."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 10 ** 6), (8, 1, 10 ** 5), (2, 2, 3 * 10 ** 5), (1, 2, 123457), (70, 1, 20011), (10, 10, 10 ** 6), (3, 4, 200003)]


@pytest.mark.parametrize("together", [False, True])
def test_long_k(together):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from trim_gb300 import uni10 as tu

    tu.set_stream(torch.cuda.current_stream().cuda_stream)
    rng = np.random.default_rng(31)
    for shapes in ([SHAPES + [(64, 64, 64)]] if together else [[s] for s in SHAPES]):
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
            assert np.all(err <= 2 * (k + 1) * 2.0 ** -53 * (np.abs(x) @ np.abs(y))), (m, n, k)


def test_sums_stay_short_in_large_lists():
    """Equal products round the same way at every step, so a sum's error grows
    with its length: with sums of 1024 products, and sums of those, it stays
    within (1024 + K / 1024 + 256) 2^-53 (relative; 1.1 rounds to 1937 of these units
    in sums of 13400).  Beside it few outputs, whose lanes hold several ranges, and
    rows."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fractions import Fraction
    from trim_gb300 import uni10 as tu

    tu.set_stream(torch.cuda.current_stream().cuda_stream)
    gemms, ao, bo, co = [], 0, 0, 0
    k = 100000
    for m, n in [(1000, 1000), (9, 10), (3, 2)]:
        gemms.append((m, n, k, ao, bo, co))
        ao, bo, co = ao + m * k, bo + k * n, co + m * n
    A = torch.ones(ao, dtype=torch.float64, device="cuda")
    B = torch.full((bo,), 1.1, dtype=torch.float64, device="cuda")
    C = torch.full((co,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    tu.contract_sectors("fp64", gemms, A.data_ptr(), B.data_ptr(), C.data_ptr())
    tu.sync()
    want = Fraction(1.1) * k
    worst = max(abs(Fraction(v) - want) / want for v in set(C.cpu().tolist()))
    assert worst <= Fraction(1024 + k // 1024 + 256, 2 ** 53)


def test_sums_stay_short_through_views():
    """The same with A read through a view of its unpermuted source."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from fractions import Fraction
    from trim_gb300 import uni10 as tu
    from trim_gb300 import workloads as wl

    tu.set_stream(torch.cuda.current_stream().cuda_stream)
    m, n, k0, k1 = 800, 800, 2, 60000  # two segments of 60000 k where the view has them
    a = tu.UniTensor([wl.dense_bond(wl.IN, m), wl.dense_bond(wl.IN, k0), wl.dense_bond(wl.IN, k1)], [0, 1, 2])
    b = tu.UniTensor([wl.dense_bond(wl.IN, k0), wl.dense_bond(wl.IN, k1), wl.dense_bond(wl.OUT, n)], [1, 2, 3])
    a.set_elem(np.ones(m * k0 * k1))
    b.set_elem(np.full(n * k0 * k1, 1.1))
    c = tu.contract(a, b).get_elem()
    want = Fraction(1.1) * k0 * k1
    worst = max(abs(Fraction(float(v)) - want) / want for v in set(c.tolist()))
    assert worst <= Fraction(1024 + k0 * k1 // 1024 + 256, 2 ** 53)
