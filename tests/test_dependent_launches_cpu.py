"""Kernels that start while the kernel before them runs (launch_dependent): the pointers to what that kernel writes
carry no __restrict__, which would promise that the data do not change while the kernel runs."""
import glob
import os
import re

from photonprop_b200 import _build

# launched as a dependent -> the parameters or members that the kernels before it on the stream write
WRITTEN_BEFORE = {
    "batched_kernel": ("RunParams", ["granule_offsets", "queue", "counters", "stats", "hist"]),
    "train_kernel": (None, ["part", "grad"]),
    "adam_kernel": (None, ["g"]),
    "llh_kernel": (None, ["chunk_start", "llh"]),
    "setup_kernel": (None, []),  # follows fill_kernel, whose outputs it is not given
}


def _sources():
    src = {}
    for f in sorted(glob.glob(os.path.join(_build.CSRC, "*.cu*"))):
        with open(f) as h:
            src[os.path.basename(f)] = re.sub(r"//[^\n]*", "", h.read())
    return src


def test_every_dependent_kernel_is_listed():
    names = set()
    for text in _sources().values():
        for m in re.finditer(r"launch_dependent\(\s*([\w:]+)", text):
            names.add(m.group(1).split("::")[-1])
    assert names - {"fn"} == set(WRITTEN_BEFORE) - {"batched_kernel"}


def test_no_restrict_on_what_the_predecessor_writes():
    text = "\n".join(_sources().values())
    for kernel, (holder, params) in WRITTEN_BEFORE.items():
        if holder:
            decl = re.search(r"struct %s \{(.*?)\n\};" % holder, text, re.S).group(1).split(";")
        else:
            decl = re.search(r"__global__[^;{]*?\b%s\(([^{]*)\)\s*\{" % kernel, text, re.S).group(1).split(",")
        for p in params:
            own = [d for d in decl if re.search(r"\*.*\b%s\s*$" % p, d.strip())]
            assert len(own) == 1, (kernel, p, own)
            assert "__restrict__" not in own[0], (kernel, p)
