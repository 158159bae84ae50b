"""The batched kernel's queue lookup: lane 0 rewrites the warp's run and flushes its statistics, which every lane has
read (and added to) without a barrier since, so the lookup begins with one; and it ends with one, before the lanes
read the new run."""
import os
import re

from photonprop_b200 import _build


def _fetch_body():
    with open(os.path.join(_build.CSRC, "pp_kernels.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    start = text.index("auto fetch = [&]() {") + len("auto fetch = [&]() {")
    depth, at = 1, start
    while depth:
        depth += {"{": 1, "}": -1}.get(text[at], 0)
        at += 1
    return [s.strip() for s in text[start:at - 1].strip().split("\n") if s.strip()]


def test_lookup_is_between_two_warp_barriers():
    body = _fetch_body()
    assert body[0] == "__syncwarp();"
    assert body[-2:] == ["__syncwarp();", "return p >= 0;"]
