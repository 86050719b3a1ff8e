"""The tile walk of permutes whose rows stay contiguous (the last bond in
place), on the CPU: rows around 32 elements, where the second tile dimension is
chosen by how well it fills the tile, next to bonds of 1, 2 and 3, for 8- and
16-byte elements, against a numpy transpose."""
import itertools

import numpy as np
import pytest

from trim_gb300 import uni10 as tu
from trim_gb300 import workloads as wl

ROWS = [1, 2, 31, 32, 33, 64, 257, 2049, 4100]
OUTER = [(2, 2, 3), (7, 2, 2), (1, 3, 40), (40, 1, 2), (9, 2, 17)]


@pytest.mark.parametrize("outer", OUTER)
@pytest.mark.parametrize("row", ROWS)
def test_row_permutes_bit_exact(row, outer):
    dims = outer + (row,)
    src = [wl.dense_bond(wl.IN if i < 2 else wl.OUT, d) for i, d in enumerate(dims)]
    n = int(np.prod(dims))
    x = np.arange(1.0, n + 1)
    for perm in itertools.permutations(range(3)):
        rsp = list(perm) + [3]
        for rn in (1, 2, 3):
            dst = [wl.change(src[b], wl.IN if j < rn else wl.OUT) for j, b in enumerate(rsp)]
            want = x.reshape(dims).transpose(rsp).ravel()
            got, written = tu.plan_check_permute(tu.SectorMap(src), tu.SectorMap(dst), rsp, x)
            assert written == n and np.array_equal(got, want)
            z = x - 2j * x
            got, written = tu.plan_check_permute_c128(tu.SectorMap(src), tu.SectorMap(dst), rsp, z)
            assert written == n and np.array_equal(got, want - 2j * want)
