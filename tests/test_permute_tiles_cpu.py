"""The tile walk of permutes with bonds between the tile sizes, on the CPU:
rows that stay in place and fill a sixteenth to a half of a tile with the bond
before them (repeated along a third bond), and transposes whose bonds are a
little over 64 (cut into equal, narrower tiles), for 8- and 16-byte elements,
against a numpy transpose."""
import itertools

import numpy as np
import pytest

from trim_gb300 import uni10 as tu
from trim_gb300 import workloads as wl

DIMS = [(5, 9, 24, 24), (24, 7, 11, 17), (3, 50, 2, 30), (2, 3, 40, 65), (9, 65, 70), (96, 2, 100), (81, 130, 3), (33, 64, 5, 16),
        (8, 4, 8, 32), (2, 67, 2, 129), (3, 2, 1000), (2, 5, 3, 700),
        (20, 3, 700, 2), (7, 40, 300, 3), (3, 4, 5, 6, 7), (2, 7, 2, 9, 10), (4, 4, 4, 4, 4, 4),
        (9000, 2), (4100, 3), (333, 31), (65, 32), (700, 63), (5, 64)]


@pytest.mark.parametrize("dims", DIMS)
def test_permutes_bit_exact(dims):
    k = len(dims)
    src = [wl.dense_bond(wl.IN if i < 2 else wl.OUT, d) for i, d in enumerate(dims)]
    n = int(np.prod(dims))
    x = np.arange(1.0, n + 1)
    for perm in itertools.permutations(range(k)):
        dst = [wl.change(src[b], wl.IN if j < 2 else wl.OUT) for j, b in enumerate(perm)]
        want = x.reshape(dims).transpose(perm).ravel()
        got, written = tu.plan_check_permute(tu.SectorMap(src), tu.SectorMap(dst), list(perm), x)
        assert written == n and np.array_equal(got, want)
        z = x - 2j * x
        got, written = tu.plan_check_permute_c128(tu.SectorMap(src), tu.SectorMap(dst), list(perm), z)
        assert written == n and np.array_equal(got, want - 2j * want)
