"""How far the tiled split-precision GEMM is from exact sums (numpy long double:
64 or 113 significant bits), with 2^e the power-of-two scale of a row of A or a
column of B (max < 2^e <= 2 max).

Per k and output, over 2^(ea+eb): the five dropped digit products are at most 5
256^2 2^-70 = 2^-51.7, and independent with a root mean square of 2^-54.4 (two
uniform digits of 512 values: 148^2 2^-70 sqrt 5) on entries without structure;
the operands' rounding is at most 2^-53 (2^-54.8 of one times the other).
So the error is below K 2^-51 2^(ea+eb) for any input and, in the Frobenius norm
and with a factor 2 for the sample, below sqrt(K) 2^-53.4 2^(ea+eb) for Gaussian
ones; the FP64 partial sums and the result add at most 2^-51 |C|.

Lists of split precision whose sectors lie on both sides of the line between
the tensor cores and the FP64 kernel: the same bound."""
import numpy as np
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


def _scales(x, axis):
    return np.ldexp(1.0, np.frexp(np.abs(x).max(axis))[1])


def _product(torch, tu, mode, work):
    gemms, ao, bo, co = [], 0, 0, 0
    for a, b in work:
        (m, k), n = a.shape, b.shape[1]
        gemms.append((m, n, k, ao, bo, co))
        ao, bo, co = ao + m * k, bo + k * n, co + m * n
    A = torch.from_numpy(np.concatenate([a.ravel() for a, _ in work])).cuda()
    B = torch.from_numpy(np.concatenate([b.ravel() for _, b in work])).cuda()
    C = torch.full((co,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    tu.contract_sectors(mode, gemms, A.data_ptr(), B.data_ptr(), C.data_ptr())
    tu.sync()
    c = C.cpu().numpy()
    return [c[off:off + m * n].reshape(m, n) for m, n, _, _, _, off in gemms]


# K = 30000 has its images made in two launches, the others in one
@pytest.mark.parametrize("m, n, k", [(33, 40, 300), (48, 33, 2000), (24, 32, 4097), (17, 20, 30000)])
def test_gaussian(env, m, n, k):
    rng = np.random.default_rng(5)
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    c, = _product(*env, "split_tiled", [(a, b)])
    exact = a.astype(np.longdouble) @ b.astype(np.longdouble)
    unit = np.outer(_scales(a, 1), _scales(b, 0))
    err = np.linalg.norm((c - exact).astype(float))
    assert err <= np.sqrt(k) * 2.0 ** -53.4 * np.linalg.norm(unit) + 2.0 ** -51 * np.linalg.norm(c)


def _of_digits(d):
    return sum(x * 2.0 ** (-8 - 9 * s) for s, x in enumerate(d))


@pytest.mark.parametrize("k", [64, 4096, 4200])
@pytest.mark.parametrize("digits", [(256, 0, 0, 0, 0, -1), (255, 255, 255, 255, 255, 255), (255, -256, -256, -256, -256, -256),
                                    (128, 255, -256, 255, -256, 255)])
def test_largest_digits(env, digits, k):
    x = _of_digits(digits)
    a, b = np.full((130, k), x), np.full((k, 65), x)
    a[1::2] = -x
    b[:, 2::3] = -x
    c, = _product(*env, "split_tiled", [(a, b)])
    exact = np.sign(a[:, :1]) * np.sign(b[:1]) * (np.longdouble(x) * np.longdouble(x) * k)
    bound = k * 2.0 ** -51 * np.outer(_scales(a, 1), _scales(b, 0)) + 2.0 ** -51 * np.abs(c)
    assert np.all(np.abs((c - exact).astype(float)) <= bound)


def test_list_of_small_and_large_sectors(env):
    rng = np.random.default_rng(9)
    shapes = [(8, 30, 900), (30, 30, 900), (12, 16, 64), (16, 16, 16), (64, 64, 40), (1, 200, 500), (200, 17, 120), (130, 70, 700),
              (15, 33, 2500), (40, 15, 300), (128, 64, 16)]
    work = [(rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (k, n))) for m, n, k in shapes]
    for (a, b), c in zip(work, _product(*env, "split", work)):
        k = a.shape[1]
        bound = k * 2.0 ** -51 * np.outer(_scales(a, 1), _scales(b, 0)) + k * 2.0 ** -52 * (np.abs(a) @ np.abs(b))
        assert np.all(np.abs((c - a.astype(np.longdouble) @ b.astype(np.longdouble)).astype(float)) <= bound)


def test_images_of_long_rows_in_one_launch(env):
    """Beside a product large enough that the images are made in one launch."""
    rng = np.random.default_rng(10)
    shapes = [(2, 22000, 1500), (12, 16, 1025), (40, 31, 1999), (9, 19, 2000), (10, 20, 2001), (6, 70, 8192)]
    work = [(rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (k, n))) for m, n, k in shapes]
    for (a, b), c in zip(work, _product(*env, "split_tiled", work)):
        k = a.shape[1]
        bound = k * 2.0 ** -51 * np.outer(_scales(a, 1), _scales(b, 0)) + k * 2.0 ** -52 * (np.abs(a) @ np.abs(b))
        assert np.all(np.abs(c - a @ b) <= bound)
