"""Blocks of a cluster meet with the aligned barrier instructions, which want every lane of a warp there together.  Read from the sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "poptransformer_b200", "csrc")


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_whole_warps_meet(path):
    """In front of every arrival stands __syncwarp(), or nothing of the kernel that lanes could take differently: only declarations."""
    text = open(path).read()
    for m in re.finditer(r'asm volatile\("barrier\.cluster\.arrive', text):
        before = re.sub(r"//[^\n]*", "", text[:m.start()]).rstrip()
        if before.endswith("__syncwarp();"):
            continue
        body = before[before.rindex("__global__"):]
        body = body[body.index(") {") + 3:]
        assert re.fullmatch(r"(\s*__shared__ [^;]*;)*\s*", body), text[m.start() - 200:m.start()]
