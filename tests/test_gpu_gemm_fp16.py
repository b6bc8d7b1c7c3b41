"""GPU parity of the fp16 product (pt_gemm, PT_W_FP16) and of k-slices that meet in a cluster, at the edges of tiles, k-slices and epilogues, against
sums in float64.  Bound: one fp16 rounding of the result (2^-11) plus what k fp32 additions of exact products lose."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(y, exp, x, w, k):
    slack = float(k * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T).max())
    assert float(((y.double() - exp).abs() - exp.abs() * 2.0 ** -11).max()) <= slack + 2.0 ** -24


# 1, 9, 16, 17, 33 rows: edges of the smallest tiles; 65, 257: a second tile; 1003 and 40 outputs: a last weight tile that is partly empty
# and an odd row stride; k of one block, and of blocks that slices do not divide.
@pytest.mark.parametrize("n,k,m", [(2048, 2048, 1), (4608, 4096, 9), (1003, 64, 16), (2048, 8192, 17), (50257, 1600, 33), (40, 1088, 65), (1600, 6400, 257)])
def test_fp16_sizes(cuda, n, k, m):
    from poptransformer_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(n + k + m)
    w, x = torch.randn((n, k), device=cuda, generator=g).half() * 0.05, torch.randn((m, k), device=cuda, generator=g).half()
    res, bias = torch.randn((m, n), device=cuda, generator=g).half(), torch.randn((n,), device=cuda, generator=g).half()
    gw, exp = ops.GemmWeight(ops.W_FP16, w), x.double() @ w.double().T
    err, ws = torch.zeros(1, dtype=torch.int32, device=cuda), ops.gemm_workspace(m, n, 8, cuda)
    for ksplit in (0, 1, 5):
        kw = dict(ksplit=ksplit, error_flag=err, workspace=ws)
        y = ops.gemm(x, gw, **kw)
        _check(y, exp, x, w, k)
        assert torch.equal(ops.gemm(x, gw, epilogue=ops.EPI_BIAS, bias=bias, **kw), y + bias)
        assert torch.equal(ops.gemm(x, gw, epilogue=ops.EPI_RESIDUAL, residual=res, **kw), res + y)
        assert torch.equal(ops.gemm(x, gw, epilogue=ops.EPI_BIAS_RESIDUAL, bias=bias, residual=res, **kw), res + (y + bias))
        z = (y + bias).double()
        gelu = ops.gemm(x, gw, epilogue=ops.EPI_BIAS_GELU, bias=bias, **kw).double()
        want = torch.nn.functional.gelu(z)
        assert bool(((gelu - want).abs() <= want.abs() * 2.0 ** -10 + z.abs() * 2.0 ** -22 + 2.0 ** -24).all())     # one fp16 rounding of a float32 value
    assert int(err.item()) == 0


@pytest.mark.parametrize("f,k,m", [(1024, 2048, 9), (504, 512, 40)])
def test_fp16_swiglu(cuda, f, k, m):
    from poptransformer_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(f + m)
    w, x = torch.randn((2 * f, k), device=cuda, generator=g).half() * 0.05, torch.randn((m, k), device=cuda, generator=g).half()
    gw, plain = ops.GemmWeight(ops.W_FP16, w, interleave_gate_up=True), ops.GemmWeight(ops.W_FP16, w)
    for ksplit in (0, 1):
        gate, up = ops.gemm(x, plain, ksplit=ksplit).float().chunk(2, 1)
        want = up.half() * torch.nn.functional.silu(gate).half()
        assert torch.allclose(ops.gemm(x, gw, epilogue=ops.EPI_SWIGLU, ksplit=ksplit).float(), want.float(), rtol=2.0 ** -9, atol=2.0 ** -24)


@pytest.mark.parametrize("n,k,m", [(4096, 13696, 8), (1003, 256, 17), (640, 4096, 64)])
def test_fp8_slices_need_no_workspace(cuda, n, k, m):
    from poptransformer_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(n + k + m)
    w8, x8 = ((torch.randn(s, device=cuda, generator=g) * 20).to(torch.float8_e4m3fn) for s in ((n, k), (m, k)))
    y = ops.gemm(x8.view(torch.uint8), ops.GemmWeight(ops.W_FP8, w8.view(torch.uint8), w_scale=2.0 ** -9), x_scale=2.0 ** -6)
    w, x = w8.float(), x8.float()
    exp = (x.double() @ w.double().T) * 2.0 ** -15
    slack = float(k * 2.0 ** -24 * 2.0 ** -15 * (x.double().abs() @ w.double().abs().T).max())
    assert float(((y.double() - exp).abs() - exp.abs() * 2.0 ** -11).max()) <= slack + 2.0 ** -24


@pytest.mark.parametrize("rows,dim", [(1, 8191), (1, 8192), (3, 50257), (33, 32000), (2, 8200)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_largest_of_a_row(cuda, rows, dim, dtype):
    """The lowest index among equals, infinities included, whatever part of the row they are in."""
    from poptransformer_b200 import ops
    x = torch.randint(-40, 40, (rows, dim), device=cuda).to(dtype)          # many equals
    x[0, :] = float("-inf")
    if rows > 1:
        x[1, dim - 1] = 100.0
    if rows > 2:
        x[2, dim // 2] = x[2, dim - 3] = float("inf")
    v, i = ops.topk(x, 1)
    first = (x == x.max(1, keepdim=True).values).int().argmax(1)
    assert torch.equal(i.view(-1).long(), first) and torch.equal(v.view(-1), x.max(1).values)
