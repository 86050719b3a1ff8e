"""The flat FP64 work list at sizes where it could grow or shrink too far, on
the CPU: dot products and few outputs over a long K are spread over the chip,
and large outputs over a long K are not cut into more items and partial sums
than the chip has use for."""
import os
import subprocess

import pytest

from tests.test_cpp_driver import LIBDIR, ROOT, shutil

SMS = 152


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(LIBDIR, "libtrim_gb300.so")):
        pytest.skip("no g++ or library not built")
    exe = str(tmp_path_factory.mktemp("flat") / "flat_plan_check")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    p = subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "trim_gb300", "csrc"), "-I" + os.path.join(cuda, "include"),
                        os.path.join(ROOT, "tests", "cpp", "flat_plan_check.cpp"), "-L" + LIBDIR, "-ltrim_gb300", "-L" + os.path.join(cuda, "lib64"),
                        "-lcudart", "-Wl,-rpath," + LIBDIR, "-Wl,-rpath," + os.path.join(cuda, "lib64"), "-o", exe], capture_output=True, text=True)
    assert p.returncode == 0, p.stderr

    def run(*shapes):
        out = subprocess.run([exe, str(SMS), *[str(v) for s in shapes for v in s]], capture_output=True, text=True).stdout.split()
        assert out and out[0] == "ok", out
        return [int(v) for v in out[1:]]

    return run


@pytest.mark.parametrize("shape", [(1, 1, 10 ** 6), (8, 1, 10 ** 5), (2, 2, 3 * 10 ** 5), (1, 2, 10 ** 8)])
def test_rows_over_a_long_k(plan, shape):
    """No warp takes more than two items' share: twice a 24th of a
    sub-partition's (64 warp FMAs at least), or a 1024th of a row."""
    m, n, k = shape
    items, _, cost, ranges, _ = plan(shape)
    share = m * n * k / 32 / (4 * SMS)
    assert cost <= max(2 * max(64, share / 24) + 5 * n, n * (k / 32 / 1024 + 2))
    assert items >= min(256, m * n * k // 4096) and ranges <= 1024


@pytest.mark.parametrize("shape", [(10, 10, 10 ** 6), (3, 4, 10 ** 6), (11, 11, 10 ** 8), (64, 1, 31)])
def test_few_outputs(plan, shape):
    _, ws, _, ranges, _ = plan(shape)
    most = max(256, 8192 // (shape[0] * shape[1]))
    assert ranges <= most and ws <= most * shape[0] * shape[1]


@pytest.mark.parametrize("shapes", [[(2800, 2800, 10 ** 5)], [(2800, 2800, 10 ** 8)], [(400, 400, 10 ** 6)] * 20, [(130, 1, 10 ** 7), (1000, 1000, 50000)], [(576, 576, 331776)], [(1000, 1000, 10 ** 5)], [(10, 10, 10 ** 5), (2000, 2000, 50000)]])
def test_large_outputs_over_a_long_k(plan, shapes):
    """Items: 768 a sub-partition and twice that for rounding, and the chunks of
    128 outputs; partial sums: 128 to an item of a split chunk.  No sum of more than
    4096 products that the kernel does not break off."""
    items, ws, _, _, chain = plan(*shapes)
    chunks = sum(m * n // 128 + 1 for m, n, _ in shapes)
    assert items <= 2 * 768 * 4 * SMS + 2 * chunks
    assert ws <= 128 * 2 * 768 * 4 * SMS
    assert chain <= 4096


@pytest.mark.parametrize("shapes", [[(1, 1, 562)], [(4, 4, 105)] * 2, [(3, 7, 14786)], [(4460, 1, 59)], [(281, 1, 55)] * 100, [(2, 39, 895)], [(9, 16, 320)] * 20])
def test_lists_that_leave_warps_idle(plan, shapes):
    """The longest item costs at most two of the least (64 warp FMAs), and a
    warp adds up no more ranges than the square root of K, or 8, unless the lanes
    run along them."""
    items, _, cost, ranges, _ = plan(*shapes)
    m, n, k = shapes[0]
    assert cost <= 2 * 64
    assert ranges <= max(8, k ** 0.5) or n <= 8 or m * n >= 128
    if n <= 8 and k >= 32:  # rows: spread over the resident warps, four to a warp at most beyond that
        rows = m * len(shapes)
        assert items >= min(rows, rows // 12)


def test_every_product_once(plan):
    plan(*[(m, n, k) for m in (1, 3, 33, 130) for n in (1, 2, 3, 32) for k in (1, 31, 32, 700, 40001)])
    plan((5, 2, 99999), (1, 1, 12345678), (7, 18, 5000), (300, 300, 64))
