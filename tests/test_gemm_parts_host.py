"""Products that share a launch: rows and outputs that do not fit are refused before a pointer is taken (the kernel writes m rows of every part)."""
import types

import pytest
import torch

from poptransformer_b200 import ops
from poptransformer_b200._lib import PtError

WEIGHT = types.SimpleNamespace(k_in=64, n_out=256)


def _out(*shape, dtype=torch.float16):
    return torch.empty(shape, dtype=dtype)


@pytest.mark.parametrize("rows,outs,why", [
    (7, [_out(3, 128), _out(3, 128)], "equal runs"),
    (8, [_out(4, 128), _out(3, 128)], r"float16 \[4, n\]"),
    (8, [_out(5, 128), _out(4, 128)], r"float16 \[4, n\]"),
    (8, [_out(4, 128), _out(4, 128, dtype=torch.float32)], r"float16 \[4, n\]"),
    (8, [_out(4, 128), _out(4 * 128)], r"float16 \[4, n\]"),
])
def test_parts_that_do_not_fit(rows, outs, why):
    with pytest.raises(PtError, match=why):
        ops.gemm(torch.empty((rows, 64), dtype=torch.float16), WEIGHT, parts=[(o, ops.EPI_STORE) for o in outs])


def test_parts_that_fit_come_to_the_pointers():
    with pytest.raises(PtError, match="CUDA tensors"):
        ops.gemm(torch.empty((8, 64), dtype=torch.float16), WEIGHT, parts=[(_out(4, 128), ops.EPI_STORE)] * 2)
