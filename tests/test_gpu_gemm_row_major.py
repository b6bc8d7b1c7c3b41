"""pt_gemm on row-major FP8 weights (a plain product of two matrices) asked to start early: what it gives without."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


# k of four and of more blocks than a ring has stages; one slice and several
@pytest.mark.parametrize("n,k,m,ksplit", [(300, 512, 16, 1), (1003, 4096, 40, 1), (1003, 4096, 40, 4), (256, 640, 200, 0)])
def test_early_start_changes_nothing(cuda, n, k, m, ksplit):
    from poptransformer_b200 import _lib, ops
    g = torch.Generator(device=cuda).manual_seed(n + k)
    w, x = ((torch.randn(s, device=cuda, generator=g) * 20).to(torch.float8_e4m3fn) for s in ((n, k), (m, k)))
    xd, wd = x.float().double(), w.float().double()
    exp = (xd @ wd.T) * 2.0 ** -15
    ws, err = ops.gemm_workspace(m, n, 8, cuda), torch.zeros(1, dtype=torch.int32, device=cuda)
    outs = []
    for pdl in (0, 1):
        a = _lib.GemmArgs()
        w8, out = torch.zeros((n, k), dtype=torch.uint8, device=cuda), torch.zeros((m, n), dtype=torch.float16, device=cuda)
        a.wfmt, a.m, a.n_out, a.k_in, a.epilogue, a.ksplit, a.w_tiled = ops.W_FP8, m, n, k, ops.EPI_STORE, ksplit, 0
        a.x, a.w, a.out = x.data_ptr(), w8.data_ptr(), out.data_ptr()
        a.x_scale, a.w_scale, a.pdl = 2.0 ** -6, 2.0 ** -9, pdl
        a.workspace, a.workspace_bytes, a.error_flag = ws.data_ptr(), ws.numel(), err.data_ptr()
        w8.copy_(w.view(torch.uint8))                 # the launch in front of the product writes its weights
        ops.check(_lib.lib().pt_gemm(ctypes.byref(a), ops._stream()), "pt_gemm")
        outs.append(out)
    assert int(err.item()) == 0 and torch.equal(*outs)
    slack = float(k * 2.0 ** -24 * 2.0 ** -15 * (xd.abs() @ wd.abs().T).max())       # k fp32 additions, one fp16 rounding
    assert float(((outs[0].double() - exp).abs() - exp.abs() * 2.0 ** -11).max()) <= slack + 2.0 ** -24
