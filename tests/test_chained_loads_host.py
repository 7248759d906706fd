"""The rule of csrc/chain.cuh for chained kernels, on the source: a read-only
load may move above the wait for the preceding kernel unless its address comes
from data loaded behind it, so no gather takes the slot's own index i (list
padding, a loaded value, may be it)."""
import importlib
import os
import re


def test_no_gather_at_the_own_index():
    build = importlib.import_module("xpbi-webgpu_gb300.build")
    with open(os.path.join(build.CSRC, "solve.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    assert "gather(j" in text  # the pair loops are still written this way
    bad = re.findall(r"gather\w*\(i\)|\bldg\([^()]*\+ i\)|make_uint2\(i, i\)", text)
    # a partner index that falls back to i and is then gathered
    for name in re.findall(r"(\w+) = [^;?]*\? sub[.\->]+\w+\([^;]*\) : i;", text):
        bad += re.findall(rf"gather\({name}\)", text)
    assert not bad, bad
