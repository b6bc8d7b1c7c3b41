"""Products in k-slices, whose sums are sent to the block that writes them or fetched by it, in every format and epilogue and at ragged sizes, against float64."""
import pytest
import torch

from poptransformer_b200 import ops

pytestmark = pytest.mark.gpu

# rows and k for: sums sent in tiles of 16 and 32 rows, fetched in tiles of 32, 48 and 64, and in several tiles of rows
SIZES = [(12, 4096), (30, 4096), (30, 1024), (45, 4096), (64, 1024), (130, 4096)]


def _weight(fmt, n, k, g, dev):
    """A tiled weight matrix and its exact values."""
    if fmt == "int4":
        gw = ops.GemmWeight(ops.W_INT4, torch.randint(-128, 128, (n, k // 2), generator=g, dtype=torch.int8, device=dev), torch.rand((n, k // 128), generator=g, device=dev).half() * 0.02, group=128)
        return gw, ops.gemm(torch.eye(k, dtype=torch.float16, device=dev), gw).T.double()
    w = torch.randn((n, k), generator=g, device=dev) * 0.05
    if fmt == "fp8":
        w8 = (w * 16).to(torch.float8_e4m3fn)
        return ops.GemmWeight(ops.W_FP8, w8.view(torch.uint8), w_scale=0.0625), w8.double() * 0.0625
    w = w.to(torch.float16 if fmt == "fp16" else torch.bfloat16)
    return ops.GemmWeight(ops.W_FP16 if fmt == "fp16" else ops.W_BF16, w), w.double()


def _rows(fmt, m, k, g, dev):
    x = torch.randn((m, k), generator=g, device=dev)
    if fmt == "fp8":
        x = x.to(torch.float8_e4m3fn)
        return x.view(torch.uint8), x.double()
    x = x.to(torch.bfloat16 if fmt == "bf16" else torch.float16)
    return x, x.double()


def _close(got, exp, size, k, roundings, most):
    """`roundings` of values up to `most` larger than the result, and k sums of which each step may lose 2^-23 of what has gathered."""
    bound = roundings * (exp.abs() + most) + size * k * 2.0 ** -23
    assert bool(((got.double() - exp).abs() <= bound).all()), float(((got.double() - exp).abs() / bound).max())


@pytest.mark.parametrize("m,k", SIZES)
@pytest.mark.parametrize("n", [203, 272])
@pytest.mark.parametrize("fmt,epilogue", [(f, e) for f in ("fp16", "int4", "fp8") for e in ("store", "residual", "bias", "swiglu", "bias_residual", "bias_gelu", "relu2", "gated_residual")
                                          if f == "fp16" or e in ("store", "residual", "bias") or (f == "int4" and e == "swiglu")])
def test_fp16_outputs(cuda, fmt, epilogue, n, m, k):
    if epilogue == "swiglu" and n % 16:
        pytest.skip("gates and ups come in blocks of eight")
    g = torch.Generator(device=cuda).manual_seed(m + n + k)
    gw, W = _weight(fmt, n, k, g, cuda)
    x, X = _rows(fmt, m, k, g, cuda)
    rand = lambda *s: torch.randn(s, generator=g, device=cuda).half()
    bias, res, gate = rand(n), rand(m, n), rand(m, n)
    y, size, B = X @ W.T, X.abs() @ W.abs().T, bias.double()
    exp = {"store": y, "residual": res + y, "bias": y + B, "bias_residual": res + (y + B), "bias_gelu": torch.nn.functional.gelu(y + B), "relu2": torch.relu(y) ** 2,
           "gated_residual": (res + torch.sigmoid(gate.double()) * y) / 2, "swiglu": None}[epilogue]
    if epilogue == "swiglu":
        v, s = y.view(m, -1, 2, 8), size.view(m, -1, 2, 8)
        exp = (torch.nn.functional.silu(v[:, :, 0]) * v[:, :, 1]).reshape(m, -1)
        size = (v[:, :, 0].abs() * s[:, :, 1] + v[:, :, 1].abs() * s[:, :, 0]).reshape(m, -1) * 2
    if epilogue == "relu2":
        size = 2 * torch.relu(y) * size
    out = res.clone() if "residual" in epilogue else torch.full(exp.shape, 7, dtype=torch.float16, device=cuda)
    err = torch.zeros(1, dtype=torch.int32, device=cuda)
    ops.gemm(x, gw, out=out, epilogue=getattr(ops, "EPI_" + epilogue.upper()), residual=out if "residual" in epilogue else None, bias=bias if "bias" in epilogue else None,
             gate=gate if "gated" in epilogue else None, halve=1, error_flag=err)
    most = float(y.abs().max()) + 8                                      # (what is added or multiplied last)
    _close(out, exp, size + 1, k, 4 * 2.0 ** -11, most if epilogue != "store" else 0)
    assert int(err.item()) == 0


@pytest.mark.parametrize("m,k", SIZES)
@pytest.mark.parametrize("n", [203, 272])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_bf16_weights(cuda, dtype, n, m, k):
    g = torch.Generator(device=cuda).manual_seed(m + n + k)
    gw, W = _weight("bf16", n, k, g, cuda)
    x, X = _rows("bf16", m, k, g, cuda)
    out = torch.full((m, n), 7, dtype=dtype, device=cuda)
    ops.gemm(x, gw, out=out, alpha=0.5)
    _close(out, X @ W.T / 2, X.abs() @ W.abs().T, k, 2.0 ** (-8 if dtype == torch.bfloat16 else -23), 0)


@pytest.mark.parametrize("m,k", SIZES)
@pytest.mark.parametrize("glu", ["silu", "gelu"])
def test_bf16_gated_units_and_a_second_output(cuda, glu, m, k):
    """Gated features, then outputs that leave in fp32."""
    g = torch.Generator(device=cuda).manual_seed(m + k)
    n, split = 203, 160
    w = (torch.randn((n, k), generator=g, device=cuda) * 0.05).bfloat16()
    bias = torch.randn(n, generator=g, device=cuda)
    lin = ops.DenseLinear(w, torch.bfloat16, bias=bias, split=split, glu=ops.GLU_SILU if glu == "silu" else ops.GLU_GELU, limit=7.0)
    x, X = _rows("bf16", m, k, g, cuda)
    out, out2 = torch.full((m, split // 2), 7, dtype=torch.bfloat16, device=cuda), torch.full((m, n - split), 7, dtype=torch.float32, device=cuda)
    lin(x, out, m, split // 2, epilogue=ops.EPI_GLU, out2=out2, out2_ld=n - split)
    y, size = X @ w.double().T + bias.double(), X.abs() @ w.double().abs().T + bias.double().abs()
    v, s = y[:, :split].reshape(m, -1, 2, 8), size[:, :split].reshape(m, -1, 2, 8)
    act = torch.nn.functional.silu(v[:, :, 0]) if glu == "silu" else torch.nn.functional.gelu(v[:, :, 0], approximate="tanh")
    # (the fast exponential and quotient cost a few 2^-22 of the product)
    _close(out, (act * v[:, :, 1]).reshape(m, -1), ((v[:, :, 0].abs() + 1) * s[:, :, 1] + v[:, :, 1].abs() * s[:, :, 0]).reshape(m, -1) * 2, k, 2.0 ** -8, 2.0 ** -8)
    _close(out2, y[:, split:], size[:, split:], k, 2.0 ** -23, 0)


@pytest.mark.parametrize("m", [20, 40, 130])
def test_parts(cuda, m):
    g = torch.Generator(device=cuda).manual_seed(m)
    k, widths = 2048, (128, 256, 203)
    w = [(torch.randn((n, k), generator=g, device=cuda) * 0.05).half() for n in widths]
    x = torch.randn((3, m, k), generator=g, device=cuda).half()
    outs = [torch.full((m, n), 7, dtype=torch.float16, device=cuda) for n in widths]
    ops.gemm(x.view(-1, k), ops.GemmWeight(ops.W_FP16, torch.cat(w)), parts=list(zip(outs, [ops.EPI_STORE, ops.EPI_RELU2, ops.EPI_STORE])))
    for i in range(3):
        y, size = x[i].double() @ w[i].double().T, x[i].double().abs() @ w[i].double().abs().T
        _close(outs[i], torch.relu(y) ** 2 if i == 1 else y, size * (1 + (2 * torch.relu(y) if i == 1 else 0)), k, 3 * 2.0 ** -11, 2.0 ** -11)
