"""The tiled split-precision GEMM at the edges of its tiles: K around the 64-k
tile, the 16-k step, the 4-tile period of the tensor-memory ring and the
4096-k segment, M and N around the 128 x 64 output tile and the 16-column
store group, against a numpy product in FP64.

Bound per output: with 2^e the power-of-two scales (2^e <= 2 max), the
operands' rounding (2^-53 2^e each) and the five dropped digit products (below
2^-52 2^(ea+eb) together with their partners) cost at most 6 2^-52 2^(ea+eb)
per k, the drain's rounding 2^-51 2^(ea+eb) per 64 k, the reference's own
summation 2^-53 k per k of the magnitudes it adds: K 2^-47 max|a| max|b|
covers their sum (24 2^-52 < 2^-47) up to the reference's, added to it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [
    (1, 1, 1), (129, 65, 15), (127, 63, 16), (128, 64, 17), (130, 48, 63), (5, 17, 64), (64, 16, 65),
    (256, 128, 192), (3, 200, 255), (200, 33, 256), (131, 80, 257), (128, 64, 320), (40, 24, 576),
    (16, 20, 4095), (129, 36, 4096), (33, 64, 4097), (7, 9, 8200),
]


@pytest.fixture(scope="module")
def env():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from trim_gb300 import uni10 as tu

    tu.set_stream(torch.cuda.current_stream().cuda_stream)
    return torch, tu


def _fill(kind, rng, shape):
    if kind == "uniform":
        return rng.uniform(-1, 1, shape)
    if kind == "constant":  # every digit product of a level of one sign: the largest level sums
        return np.full(shape, 1.0 - 2.0 ** -9 - 2.0 ** -18 - 2.0 ** -27 - 2.0 ** -36 - 2.0 ** -45)
    # half-way digits (+-256 in every place) of either sign
    return np.where(rng.random(shape) < 0.9, 1.0, -1.0) * (2.0 ** -8 + 2.0 ** -17 + 2.0 ** -26 + 2.0 ** -35 + 2.0 ** -44 + 0.5)


@pytest.mark.parametrize("grouped", [False, True])
@pytest.mark.parametrize("kind", ["uniform", "constant", "halfway"])
def test_split_tiled_edges(env, kind, grouped):
    torch, tu = env
    rng = np.random.default_rng(17)
    work = []
    for m, n, k in SHAPES:
        work.append((_fill(kind, rng, (m, k)), _fill(kind, rng, (k, n))))
    for batch in ([work] if grouped else [[w] for w in work]):
        gemms, ao, bo, co = [], 0, 0, 0
        for a, b in batch:
            (m, k), n = a.shape, b.shape[1]
            gemms.append((m, n, k, ao, bo, co))
            ao, bo, co = ao + m * k, bo + k * n, co + m * n
        A = torch.from_numpy(np.concatenate([a.ravel() for a, _ in batch])).cuda()
        B = torch.from_numpy(np.concatenate([b.ravel() for _, b in batch])).cuda()
        C = torch.full((co,), float("nan"), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        tu.contract_sectors("split_tiled", gemms, A.data_ptr(), B.data_ptr(), C.data_ptr())
        tu.sync()
        c = C.cpu().numpy()
        for (a, b), (m, n, k, _, _, off) in zip(batch, gemms):
            want = a @ b
            bound = k * 2.0 ** -47 * np.abs(a).max() * np.abs(b).max() + k * 2.0 ** -53 * (np.abs(a) @ np.abs(b))
            err = np.abs(c[off:off + m * n].reshape(m, n) - want)
            assert np.all(err <= bound), (kind, m, n, k, float((err / bound).max()))
