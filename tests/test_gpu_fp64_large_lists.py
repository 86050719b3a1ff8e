"""FP64 lists with a sector of 2^23 outputs or more, which take the tiled
kernel: its narrow tile widths, its rows of narrow sectors, its K ranges, and
operands read through views, against torch's FP64 product.  Any order of K
products and sums errs by at most K 2^-53 of the sum of magnitudes (to first
order), here and in the reference."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from trim_gb300 import uni10 as tu

    tu.set_stream(torch.cuda.current_stream().cuda_stream)
    return torch, tu


def test_list_with_a_large_sector(env):
    torch, tu = env
    g = torch.Generator(device="cuda").manual_seed(3)
    shapes = [(2900, 2900, 40)]  # 8.41e6 outputs
    shapes += [(m, n, k) for m in (1, 130) for n in (1, 3, 4, 5, 8, 9, 16, 17, 31, 33) for k in (1, 31, 32, 300)]
    shapes += [(3, 5, 60000), (1, 1, 9000), (17, 40, 30011)]  # K ranges
    gemms, ao, bo, co = [], 0, 0, 0
    for m, n, k in shapes:
        gemms.append((m, n, k, ao, bo, co))
        ao, bo, co = ao + m * k, bo + k * n, co + m * n
    a, b = (torch.rand(v, generator=g, dtype=torch.float64, device="cuda") * 2 - 1 for v in (ao, bo))
    outs = []
    for _ in range(2):
        c = torch.full((co,), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        tu.contract_sectors("fp64", gemms, a.data_ptr(), b.data_ptr(), c.data_ptr())
        tu.sync()
        outs.append(c)
    assert torch.equal(outs[0], outs[1])
    for m, n, k, oa, ob, oc in gemms:
        x, y = a[oa:oa + m * k].view(m, k), b[ob:ob + k * n].view(k, n)
        err = (outs[0][oc:oc + m * n].view(m, n) - x @ y).abs()
        assert bool((err <= 2 * (k + 1) * 2.0 ** -53 * (x.abs() @ y.abs())).all()), (m, n, k)


@pytest.mark.parametrize("moved", ["a", "b", "both"])
def test_large_sector_through_views(env, moved):
    torch, tu = env
    from trim_gb300 import capi
    from trim_gb300 import workloads as wl

    m, n, k = 2900, 2900, 33
    i, o = (lambda d: wl.dense_bond(wl.IN, d)), (lambda d: wl.dense_bond(wl.OUT, d))
    g = torch.Generator(device="cuda").manual_seed(4)
    x, y = (torch.rand(v, generator=g, dtype=torch.float64, device="cuda") * 2 - 1 for v in (m * k, k * n))
    # both bonds IN: the permute to (row | column) is a view
    a = tu.UniTensor([i(m), i(k)] if moved != "b" else [i(m), o(k)], [0, 1])
    b = tu.UniTensor([i(k), i(n)] if moved != "a" else [i(k), o(n)], [1, 2])
    torch.cuda.synchronize()
    capi.call("tn_tensor_set_elem_device", a.h, x.data_ptr(), x.numel())
    capi.call("tn_tensor_set_elem_device", b.h, y.data_ptr(), y.numel())
    c = torch.from_numpy(tu.contract(a, b).get_elem()).cuda().view(m, n)
    x, y = x.view(m, k), y.view(k, n)
    assert bool(((c - x @ y).abs() <= 2 * (k + 1) * 2.0 ** -53 * (x.abs() @ y.abs())).all())
