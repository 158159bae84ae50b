"""A context does without its pinned staging block where none can be had: pp_create goes on, and pp_propagate stages
only if the block is there.  (Running out of pinned memory cannot be provoked here, so this reads the source.)"""
import os
import re

from photonprop_b200 import _build


def test_no_call_depends_on_the_pinned_block():
    with open(os.path.join(_build.CSRC, "pp_capi.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    alloc = re.findall(r"if \(cudaHostAlloc\(&c->stage[^)]*\)\) \{(.*?)\}", text, re.S)
    assert len(alloc) == 1 and text.count("cudaHostAlloc(") == 1
    assert "return" not in alloc[0] and "c->stage = nullptr;" in alloc[0]
    assert re.search(r"const bool staged = c->stage &&", text)
