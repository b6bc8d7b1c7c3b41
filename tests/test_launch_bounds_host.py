"""A kernel whose block is chosen when it is launched says how many threads that may be (__launch_bounds__): the compiler then keeps its registers within what an
SM has for so many, where a launch of more would be refused.  Read from the sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "poptransformer_b200", "csrc")
CONSTANT = r"[\s\d*+/()A-Z_:a-z]*\b[A-Z][A-Z\d_]{2,}\b[\s\d*+/()A-Z_:]*|\d+|k[A-Z]\w*"


def _arguments(text, i):
    """The arguments of the call whose opening bracket is text[i]; commas of template arguments are none of the call's."""
    parts, depth, start = [], 0, i + 1
    for j in range(i, len(text)):
        c = text[j]
        depth += (c in "([{") - (c in ")]}")
        if (c == "," and depth == 1) or depth == 0:
            part = text[start:j].strip()
            if parts and parts[-1].count("<") > parts[-1].count(">"):
                parts[-1] += ", " + part
            else:
                parts.append(part)
            start = j + 1
        if depth == 0:
            return parts


def _launches(text):
    for m in re.finditer(r"launch_early\(", text):
        args = _arguments(text, m.end() - 1)
        if not args[0].startswith("void"):
            yield args[0], args[2]
    for m in re.finditer(r"([\w:]+)(<[^<>;]*>)?<<<(.*?)>>>", text):
        yield m.group(1), _arguments("(" + m.group(3) + ")", 0)[1]


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_blocks_chosen_at_launch_are_bounded(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    bounded = {m.group(2): bool(m.group(1)) for m in re.finditer(r"__global__ void (__launch_bounds__\((?:[^()]|\([^()]*\))*\) )?(\w+)\(", text)}
    for kernel, block in _launches(text):
        block = re.sub(r"^dim3\((.*)\)$", r"\1", block)
        if re.fullmatch(CONSTANT, block) and not re.search(r"std::|threads", block):
            continue
        name = re.match(r"(?:\w+::)*(\w+)", kernel).group(1)
        names = [name] if name in bounded else re.findall(r"(\w+_kernel)<", " ".join(re.findall(r"const auto %s = ([^;]*);" % name, text)))
        assert names, (kernel, block)      # (a variable stands for the kernels that it may be)
        for n in names:
            assert bounded[n], (n, block)
