"""A kernel that is launched before the kernel in front of it has ended (launch_early) has to wait for it: its first statement is early_start(), or
it says where it waits.  Read from the sources, so that no race has to be run to see it."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "poptransformer_b200", "csrc")


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_early_launches_wait(path):
    text = open(path).read()
    launched = {n for m in re.finditer(r"launch_early\(([^,]*?),", text) for n in re.findall(r"\w+_kernel", m.group(1))}
    for name in launched:
        m = re.search(r"__global__ void (?:__launch_bounds__\((?:[^()]|\([^()]*\))*\) )?%s\(" % name, text)
        assert m, name
        body = text[text.index("{", text.index(") {", m.end())):text.index("\n}\n", m.end())]
        assert "early_start();" in body or "wait_for_prerequisites();" in body, f"{name} does not wait"
