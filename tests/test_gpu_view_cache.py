"""More operand views than the view cache holds (4096), after which it starts
over: a contraction must not meet the view table of another one whose views lay
at the same address."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_more_views_than_the_cache_holds():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from trim_gb300 import uni10 as tu
    from trim_gb300 import workloads as wl

    tu.set_stream(torch.cuda.current_stream().cuda_stream)
    rng = np.random.default_rng(5)
    x = rng.uniform(-1, 1, 128 * 64)
    shapes = [(m, k) for k in range(2, 41) for m in range(2, 113)]  # 4329 of them
    for m, k in shapes + shapes[:60]:
        a = tu.UniTensor([wl.dense_bond(wl.IN, m), wl.dense_bond(wl.IN, k)], [0, 1])  # (m, k | ) -> (m | k): a view
        b = tu.UniTensor([wl.dense_bond(wl.IN, k), wl.dense_bond(wl.OUT, 2)], [1, 2])
        a.set_elem(x[:m * k])
        b.set_elem(x[-2 * k:])
        c = tu.contract(a, b)
        want = x[:m * k].reshape(m, k) @ x[-2 * k:].reshape(k, 2)
        np.testing.assert_allclose(c.get_elem().reshape(m, 2), want, rtol=0, atol=2 * (k + 1) * k * 2.0 ** -53)
