"""A kernel that is launched before the kernel in front of it has ended has to wait for it before it reads what that one wrote.  Read from the
sources, so that no race has to be run to see it.  Launched early is what goes through launch_early or sets the launch attribute itself."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "poptransformer_b200", "csrc")
WAIT = re.compile(r"(?:early_start|wait_for_prerequisites)\(\);")
ATTRIBUTE = "cudaLaunchAttributeProgrammaticStreamSerialization"

# Kernels that do something before they wait, with the fields of their parameters that this may touch: sizes, and weights, which no launch
# of a step writes.
BEFORE = {
    "kv_append_attn_kernel": {"page", "runs", "max_pages", "qpk", "qsplit"},
    "linear_kernel": {"n_rt", "chunks_per_split", "nchunks", "B", "xs_stride", "x", "w", "pdl"},     # (x: its address)
    "prep_kernel": set(),
    "absorb_kernel": {"w_k", "rank", "dim"},
    "expand_kernel": {"w_v", "vdim", "rank", "ng", "n_tok"},
    "combine_kernel": set(),
    "decode_kernel": {"row_ld", "slots", "n_head"},
}
# The GEMMs' warps have roles.  Where each of them turns to what the launch in front wrote (its first read, or the output and the residual), it has
# just waited; the third part of a pattern is what follows the wait.
ROLES = {
    "gemm_dense_kernel": [r"if \(p\.pdl\) wait_for_prerequisites\(\);[^\n]*\n\s*const int grp = p\.group_of\[",
                          r"load_w\([^\n]*\n\s*\}\n\s*wait_for_prerequisites\(\);\n\s*\}\n\s*for \(int it = 0; it < n_it; \+\+it\) \{(?:(?!\n      \}).)*?tma_load_2d\([^\n]*&map_x",
                          r"if \(p\.pdl\) wait_for_prerequisites\(\);[^\n]*\n\s*const bool done = warp_wait\(sa\(&ctl\.accum\)",
                          r"if \(p\.pdl\) wait_for_prerequisites\(\);\n\s*sum_cluster<"],
    "gemm_int4_kernel": [r"if \(p\.pdl\) wait_for_prerequisites\(\);\n(?:(?!\n    \}).)*?tma_load_2d\([^\n]*&map_x",
                         r"if \(p\.pdl\) wait_for_prerequisites\(\);[^\n]*\n\s*const bool done = warp_wait\(sa\(&ctl\.accum\)",
                         r"if \(p\.pdl\) wait_for_prerequisites\(\);\n\s*sum_cluster<"],
}


def _source(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


def _argument(text, start):
    """The argument that begins at `start`, up to a comma or bracket outside all brackets (template arguments included)."""
    depth, i = 0, start
    while not (depth == 0 and text[i] in ",)"):
        depth += {"(": 1, "<": 1, ")": -1, ">": -1}.get(text[i], 0)
        i += 1
    return text[start:i].strip()


def _kernels(text, at, arg):
    """Names of the kernels that an argument stands for: its own, or those that the variable was last set to before position `at`."""
    names = set(re.findall(r"\w+_kernel\b", arg))
    if not names:
        assert re.fullmatch(r"\w+", arg), arg
        sets = [m.group(1) for m in re.finditer(r"\bauto\s+%s\s*=\s*([^;]*);" % arg, text[:at])]
        names = set(re.findall(r"\w+_kernel\b", sets[-1])) if sets else set()
    assert names, f"which kernel is {arg}?"
    return names


def _early(text):
    names = set()
    for m in re.finditer(r"\blaunch_early\(", text):
        if not re.match(r"void \(\*kernel\)", text[m.end():]):       # (its definition)
            names |= _kernels(text, m.start(), _argument(text, m.end()))
    for m in re.finditer(ATTRIBUTE, text):
        end = text.index("\n}\n", m.start())
        function = text[text.rindex("\n}\n", 0, m.start()) if "\n}\n" in text[:m.start()] else 0:end]
        if "launch_early(void (*kernel)" in function:
            continue
        launches = [k.end() for k in re.finditer(r"cudaLaunchKernelEx\(&cfg, ", text[:end]) if k.start() > m.start()]
        assert launches, function[:200]
        for start in launches:
            names |= _kernels(text, start, _argument(text, start))
    return names


def _body(text, name):
    m = re.search(r"__global__ void (?:__cluster_dims__\([^()]*\) )?(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\) )?%s\(" % name, text)
    assert m, name
    return text[text.index("{", text.index(") {", m.end())) + 1:text.index("\n}\n", m.end())]


FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu")))


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_early_launches_wait(path):
    text = _source(path)
    for name in _early(text):
        body = _body(text, name)
        if name in ROLES:
            for pattern in ROLES[name]:
                assert re.search(pattern, body, re.S), (name, pattern)
            continue
        if name not in BEFORE:
            assert body.lstrip().startswith("early_start();"), f"{name}: the wait is not its first statement"
            continue
        # (a product with groups waits before it looks up its matrix, and again where every product waits)
        body = re.sub(r"if \(p\.group_of\) \{\n\s*if \(p\.pdl\) wait_for_prerequisites\(\);[^\n]*\n.*?\n    \}\n", "", body, flags=re.S)
        wait = WAIT.search(body)
        assert wait, f"{name} does not wait"
        touched = set(re.findall(r"\bp\.(\w+)", body[:wait.start()]))
        assert touched <= BEFORE[name], (name, touched - BEFORE[name])


def test_named_kernels_exist():
    early = set().union(*(_early(_source(p)) for p in FILES))
    assert set(BEFORE) | set(ROLES) <= early and len(early) >= 25


def test_one_way_to_launch_early():
    """The helper exists once, and the attribute is set by hand only where the launch has other attributes or a switch."""
    where = {os.path.basename(p): len(re.findall(ATTRIBUTE, _source(p))) for p in glob.glob(os.path.join(CSRC, "*.cu*"))}
    assert {k: v for k, v in where.items() if v} == {"common.cuh": 1, "attention.cu": 1, "linear.cu": 1, "gemm_tc.cu": 1}
