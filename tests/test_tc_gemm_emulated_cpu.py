"""The tiled tensor-core GEMM kernels' own source run on the CPU, a CTA at a
time, with emulated barriers, bulk copies, MMAs and tensor memory that complete
at random times (tests/cpp/cta_emulator.h): the products at ragged sizes, K
ranges and several items per CTA; and a copy or an MMA that takes longer than
the waits' limit, after which the kernel has to record the timeout and leave
with nothing in flight, every warp whole at its warp-wide instructions."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
KERNELS = os.path.join(ROOT, "trim_gb300", "csrc", "kernels")


def _without_ptx(text):
    """The text without the functions made of inline PTX (the emulator has its own)."""
    out, at = "", 0
    for m in re.finditer(r"^(?:template <[^\n]*\n)?__device__ __forceinline__[^;{]*\{", text, re.M):
        depth, end = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        if "asm volatile" in text[m.start():end] or "__cvta_" in text[m.start():end]:
            out, at = out + text[at:m.start()], end
    return out + text[at:]


def _kernel(name):
    text = open(os.path.join(KERNELS, name)).read()
    body = text[text.index("namespace tn {"):]
    body = re.sub(r"^// -+ launchers\n", "", body, flags=re.M)
    body = body[:re.search(r"^(?:template <int NS>\n)?void launch_", body, re.M).start()]
    body = body[:body.rindex("}  // namespace")] if body.rstrip().endswith("}  // namespace") else body
    body = body.replace("extern __shared__ uint8_t dyn[];", "uint8_t* dyn = ::emu::dyn;")
    body = body.replace("extern __shared__ __align__(16) double stage[];", "double* stage = (double*)::emu::dyn;")
    return "namespace " + name.split(".")[0] + "_src {}\n" + _without_ptx(body) + "}\n}\n"


def _build(d, program, *kernels):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    ptx, digits = (open(os.path.join(KERNELS, f)).read().replace("#pragma once", "") for f in ("sm103_ptx.cuh", "tc_digits.cuh"))
    (d / (program.replace("emulated.cpp", "processed.h"))).write_text('#include "engine/engine.h"\n' + _without_ptx(ptx) + digits + "".join(kernels))
    for f in ("cta_emulator.h", program):
        shutil.copy(os.path.join(ROOT, "tests", "cpp", f), d / f)
    out = str(d / "emu")
    p = subprocess.run(["g++", "-std=c++17", "-O2", "-w", "-I" + str(d), "-I" + os.path.join(ROOT, "trim_gb300", "csrc"),
                        "-I" + os.path.join(cuda, "include"), str(d / program), "-o", out], capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-4000:]
    return out


@pytest.fixture(scope="session")
def exe(tmp_path_factory):
    # the two files' anonymous constants side by side
    fast = re.sub(r"\b(kTM|kTN|kTK|kATile|kBTile|kEpiWarps|kEpiCols|kUnit|raise_timeout|warp_wait)\b", r"\1Fast", _kernel("gemm_tc_fast.cu"))
    return _build(tmp_path_factory.mktemp("emu"), "tc_gemm_emulated.cpp", _kernel("gemm_tc_split.cu"), fast)


@pytest.fixture(scope="session")
def slice_exe(tmp_path_factory):
    return _build(tmp_path_factory.mktemp("emu"), "tc_slice_emulated.cpp", _kernel("gemm_tc.cu"))


def _run(exe, *args):
    p = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=300)
    return p.stdout.strip() or "signal %d" % p.returncode


# (M, N, K, 64-k tiles per K range, column tiles per item)
SIZES = [(1, 1, 16, 99, 1), (130, 70, 100, 99, 1), (37, 129, 640, 3, 1), (128, 64, 64, 99, 1), (257, 200, 333, 99, 4), (20, 321, 90, 1, 4),
         (5, 17, 47, 99, 2)]


@pytest.mark.parametrize("size", SIZES)
# of the sum of magnitudes: BF16 and TF32 operands are rounded by 2^-9 and 2^-12
# each (and FP32 sums of 700 products by less than 2^-14), the split form's at
# 2^-54 of a row's scale, at most 2^8 times the mean of its 1 to 700 magnitudes
@pytest.mark.parametrize("mode,bound", [("split", 2.0 ** -44), ("bf16", 2.0 ** -7.9), ("tf32", 2.0 ** -10.9)])
def test_products(exe, mode, bound, size):
    out = _run(exe, mode, *size[:4], 1 if mode == "split" else size[4], 1)
    assert out.startswith("ok") and float(out.split()[1]) < bound, out


@pytest.mark.parametrize("mode", ["split", "bf16", "tf32"])
@pytest.mark.parametrize("hold", ["hold-copy", "hold-mma"])
def test_a_wait_that_gives_up(exe, mode, hold):
    for seed in range(2):
        out = _run(exe, mode, 130, 130, 700, 99, 1 if mode == "split" else 2, seed, hold, 3 + 7 * seed)
        assert out == "timeout", out


# rows and columns around the strips of 16 and the groups of 8, K around the
# staged extents (1024 a warp, 8192 a CTA) and odd, from a null base
@pytest.mark.parametrize("size", [(9, 17, 33), (1, 1, 1), (8, 16, 576), (3, 5, 1041), (9, 3, 1100), (2, 3, 1101), (2, 3, 2001), (1, 2, 8200), (20, 40, 100)])
def test_slicing_addresses(slice_exe, size):
    if size[2] > 576:  # longer strips are a cluster's
        size = (size[0], 0, size[2])
    assert _run(slice_exe, *size, 5) == "ok"
