"""The step kernels' arguments, checked in the sources.

A block waits for its first read of each 256 bytes of its arguments, so what the
staged kernels read on every launch has to stand together: the members spread
over one line more cost the FP16 cavity 0.3 us a step.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imexlb_b200", "csrc")


def test_staged_kernels_arguments_stand_together():
    with open(os.path.join(CSRC, "lattice.h")) as fh:
        text = re.search(r"struct StepArgs \{(.*?)\n\};", fh.read(), re.S).group(1)
    names = re.findall(r"(\w+)(?:\[\w+\])? = ", re.sub(r"//[^\n]*", "", text))
    at = names.index("src")
    assert sorted(names[at:at + 7]) == sorted(["src", "dst", "err", "tickets", "rec_src", "rec_dst", "wait_ns"])


def test_tile_geometry_comes_first():
    with open(os.path.join(CSRC, "kernels.cu")) as fh:
        heads = re.findall(r"\bstaged_(?:free_)?kernel\((const [^)]*)\) \{", fh.read())
    assert heads and all(h.startswith("const stage::Geo g") for h in heads)
