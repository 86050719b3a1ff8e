"""Instructions that want a whole warp (.sync.aligned) or count whole warps (the
cluster barrier) stand in helper functions that bring the warp together first:
a CTA barrier or the end of a divergent loop does not."""
import glob
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
WIDE = re.compile(r"\.sync\.aligned|barrier\.cluster\.arrive")


def helpers():
    for p in sorted(glob.glob(os.path.join(ROOT, "trim_gb300", "csrc", "kernels", "*.cu*"))):
        text = open(p).read()
        for m in re.finditer(r"^__device__ __forceinline__[^;{]*?(\w+)\([^;{]*\{", text, re.M):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            body = re.sub(r"//.*", "", text[m.end():end])
            if WIDE.search(body):
                yield os.path.basename(p), m.group(1), body


def test_every_warp_wide_instruction_is_in_a_helper():
    inside = sum(len(WIDE.findall(body)) for _, _, body in helpers())
    files = glob.glob(os.path.join(ROOT, "trim_gb300", "csrc", "kernels", "*.cu*"))
    everywhere = sum(len(WIDE.findall(re.sub(r"//.*", "", open(p).read()))) for p in files)
    assert inside == everywhere > 0


@pytest.mark.parametrize("where", list(helpers()), ids=lambda h: h[1])
def test_the_warp_is_whole_there(where):
    name, helper, body = where
    first = min(m.start() for m in WIDE.finditer(body))
    if "__syncwarp()" not in body[:first]:  # then every call stands right behind a warp-wide vote
        text = re.sub(r"//.*", "", open(os.path.join(ROOT, "trim_gb300", "csrc", "kernels", name)).read())
        calls = len(re.findall(r"(?<!void )\b%s\(" % helper, text))
        voted = len(re.findall(r"warp_wait\([^;]*\)\) \{\s*ok = false;\s*break;\s*\}\s*tc_fence_after\(\);\s*float [^;]*;\s*%s\(" % helper, text))
        assert voted == calls > 0
    assert "barrier.cluster.arrive.release.aligned" not in body
