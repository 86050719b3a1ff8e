"""Planning a permute takes microseconds whatever the bonds' extents, and the
tiles are those that were measured, small plans' as small as they were."""
import os
import subprocess

import pytest

from tests.test_cpp_driver import LIBDIR, ROOT, shutil


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(LIBDIR, "libtrim_gb300.so")):
        pytest.skip("no g++ or library not built")
    exe = str(tmp_path_factory.mktemp("perm") / "perm_plan_check")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    p = subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "trim_gb300", "csrc"), "-I" + os.path.join(cuda, "include"),
                        os.path.join(ROOT, "tests", "cpp", "perm_plan_check.cpp"), "-L" + LIBDIR, "-ltrim_gb300", "-L" + os.path.join(cuda, "lib64"),
                        "-lcudart", "-Wl,-rpath," + LIBDIR, "-Wl,-rpath," + os.path.join(cuda, "lib64"), "-o", exe], capture_output=True, text=True)
    assert p.returncode == 0, p.stderr

    def run(order, *dims):
        out = subprocess.run([exe, order, *map(str, dims)], capture_output=True, text=True).stdout.split("\n")
        return [[float(v) for v in line.split()] for line in out if line]

    return run


@pytest.mark.parametrize("dims", [(90000000, 2), (60000000, 40), (20000000, 9), (3000000, 7), (2, 90000000)])
def test_planning_time(plan, dims):
    """A few microseconds; 5 000 is far above any noise and far below the 27 000
    to 148 000 that trying every split of such a bond took."""
    for row in plan("10", *dims):
        assert row[0] < 5000


@pytest.mark.parametrize("order,dims,tile", [("3210", (96, 96, 96, 96), (1, 32, 96)), ("10", (3000000, 3), (1, 1364, 3)),
                                             ("10", (64, 64), (1, 64, 64)), ("10", (100, 100), (1, 64, 64)), ("10", (3000, 3), (1, 64, 3)),
                                             ("32140", (2, 59, 14, 6, 5), (2, 2, 5)), ("231045", (2, 16, 15, 9, 5, 7), (3, 35, 2)),
                                             ("021", (133, 133, 133), (1, 64, 64)), ("10", (329579, 212), (1, 64, 64))])
def test_tiles(plan, order, dims, tile):
    mode, tx, ty = plan(order, *dims)[0][1:4]
    assert (mode, tx, ty) == tile
