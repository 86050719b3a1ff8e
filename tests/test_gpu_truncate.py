"""Global truncation on either side of what one CTA searches in shared memory
(about 27 000 values), with ties, zeros of both signs, empty sectors, and chi
from nothing to everything, against the oracle: the kept counts are equal and,
both norms being sums of the same non-negative squares, the norm and the scaled
values agree within (total + 8) 2^-53 relative."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[1], [5, 0, 3, 1], [60] * 25, [700, 0, 1, 900, 333], [26000, 40, 900], [9000, 9000, 12001]])
def test_truncate(sizes):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from oracle import symtensor as st
    from trim_gb300 import uni10 as tu

    tu.set_stream(torch.cuda.current_stream().cuda_stream)
    rng = np.random.default_rng(len(sizes))
    vals = [np.sort(rng.integers(0, 400, n) / 64.0)[::-1].copy() for n in sizes]  # ties within and between sectors
    for v in vals:
        v[(v == 0) & (rng.random(len(v)) < 0.5)] = -0.0
    total, off = sum(sizes), np.concatenate([[0], np.cumsum(sizes)[:-1]]).tolist()
    for chi in sorted({0, 1, total // 3, total - 1, total, total + 5}):
        S = torch.from_numpy(np.concatenate(vals)).cuda()
        torch.cuda.synchronize()
        kept, norm = tu.truncate_sectors(off, sizes, S.data_ptr(), chi)
        tu.sync()
        k_ref, n_ref, s_ref = st.truncate_global(vals, chi)
        assert list(kept) == list(k_ref), (chi, kept, k_ref)
        tol = (total + 8) * 2.0 ** -53
        assert abs(norm - n_ref) <= tol * n_ref
        got = S.cpu().numpy()
        for o, k, v, r in zip(off, kept, vals, s_ref):
            if n_ref > 0:
                np.testing.assert_allclose(got[o:o + k], np.asarray(r[:k]), rtol=2 * tol)
            assert np.array_equal(got[o + k:o + len(v)], v[k:])
