"""GPU parity of the INT4 product (pt_gemm, PT_W_INT4) at the sizes where its tiles, k-slices and epilogues change: against the products of
the dequantised fp16 weights (oracle.ops_np.int4_to_half) summed in float64.  The bound is one fp16 rounding of the result (2^-11
relative; SwiGLU: three, of both sums and of the product) plus what k fp32 additions of exact products lose (k 2^-24 of their
absolute values' sum, which the largest output bounds from below by a factor of about sqrt(k))."""
import numpy as np
import pytest
import torch

from oracle import ops_np as O

pytestmark = pytest.mark.gpu


def _case(n, k, group, m, cuda):
    r = np.random.default_rng(n + 3 * k + m)
    packed = r.integers(-128, 128, size=(n, k // 2), dtype=np.int8)
    scale = (r.random((n, k // group), dtype=np.float32) * 0.004 + 0.004).astype(np.float16)
    x = r.standard_normal((m, k), dtype=np.float32).astype(np.float16)
    w = torch.from_numpy(O.int4_to_half(packed, scale, axis=1, group=group)).to(cuda).double()
    xd = torch.from_numpy(x).to(cuda)
    return torch.from_numpy(packed).to(cuda), torch.from_numpy(scale).to(cuda), xd, xd.double() @ w, float(k * 2.0 ** -24 * (xd.double().abs() @ w.abs()).max())


# 1 / 15 / 16 / 17 rows: edges of the smallest tile; 129, 256, 257: of the tile for two CTAs per SM and of the largest; 511, 1024: prompts, whose tiles
# of 176 and 256 rows have fewer slots than the smaller ones.
# 1000 and 40 outputs: a last weight tile that is partly empty, an odd number of groups along k, a k too short for slices.
@pytest.mark.parametrize("n,k,group,m", [(4096, 4096, 128, 1), (1000, 512, 256, 15), (4096, 11008, 128, 16), (12288, 4096, 4096, 17), (40, 128, 128, 33),
                                         (1000, 1152, 384, 129), (2048, 2048, 128, 256), (1008, 1024, 128, 257), (4096, 4096, 128, 511), (12288, 1536, 128, 511), (4096, 2048, 128, 1024)])
def test_int4_sizes(cuda, n, k, group, m):
    from poptransformer_b200 import ops
    w, sc, x, exp, slack = _case(n, k, group, m, cuda)
    gw, ws, err = ops.GemmWeight(ops.W_INT4, w, sc, group=group), ops.gemm_workspace(m, n, 8, cuda), torch.zeros(1, dtype=torch.int32, device=cuda)
    res = torch.randn((m, n), device=cuda).half()
    bias = torch.randn((n,), device=cuda).half()
    for ksplit in (0, 1, 2, 7):
        kw = dict(workspace=ws, ksplit=ksplit, error_flag=err)
        y = ops.gemm(x, gw, **kw)
        assert float(((y.double() - exp).abs() - exp.abs() * 2.0 ** -11).max()) <= slack + 2.0 ** -24
        assert torch.equal(ops.gemm(x, gw, epilogue=ops.EPI_RESIDUAL, residual=res, **kw), res + y)
        assert torch.equal(ops.gemm(x, gw, epilogue=ops.EPI_BIAS, bias=bias, **kw), y + bias)
        wide = torch.full((m, n + 3), 7.0, device=cuda, dtype=torch.float16)          # an odd row stride: single stores
        assert torch.equal(ops.gemm(x, gw, out=wide, out_ld=n + 3, **kw)[:, :n], y) and float(wide[:, n:].min()) == 7.0
    assert int(err.item()) == 0


@pytest.mark.parametrize("f,k,m", [(5504, 1024, 16), (504, 512, 40), (1024, 2048, 257)])
def test_int4_swiglu(cuda, f, k, m):
    from poptransformer_b200 import ops
    w, sc, x, exp, slack = _case(2 * f, k, 128, m, cuda)
    gw, ws = ops.GemmWeight(ops.W_INT4, w, sc, group=128, interleave_gate_up=True), ops.gemm_workspace(m, 2 * f, 8, cuda)
    g, u = exp[:, :f], exp[:, f:]
    want = g / (1 + torch.exp(-g)) * u
    # |swish'| <= 1.1: what the roundings and sums of gate and up can move the product by
    bound = want.abs() * 4 * 2.0 ** -11 + (1.1 * u.abs() + g.abs()) * slack + 1.1 * u.abs() * g.abs() * 2.0 ** -11 + 1e-6
    for ksplit in (0, 1, 3):
        y = ops.gemm(x, gw, epilogue=ops.EPI_SWIGLU, workspace=ws, ksplit=ksplit)
        assert y.shape == (m, f) and bool(((y.double() - want).abs() <= bound).all())
