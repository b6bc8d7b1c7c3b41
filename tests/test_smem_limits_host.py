"""The limit of dynamic shared memory of a kernel belongs to a device: a process that works on several raises it on each.  With one GPU at hand
this is read from the sources of the attention kernels, whose tiles outgrew the default limit, and of the GEMMs, which take linears of few rows."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "poptransformer_b200", "csrc")


@pytest.mark.parametrize("name", ["attention.cu", "prefill.cu", "gemm_tc.cu"])
def test_limits_are_raised_on_every_device(name):
    text = open(os.path.join(CSRC, name)).read()
    assert "cudaFuncSetAttribute" not in text and not re.search(r"static bool", text) and "allow_smem(" in text
