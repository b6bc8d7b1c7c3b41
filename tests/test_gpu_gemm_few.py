"""Small products of up to eight activation rows at the edges of their split, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# (n, k): whole blocks and ragged ends of weight rows, one k block, warps that share k with a remainder, clusters, many rounds of blocks; the
# last two are not theirs (too large a matrix)
@pytest.mark.parametrize("n,k", [(16, 64), (40, 64), (24, 1600), (768, 768), (2056, 512), (768, 3072), (1000, 4096), (50257, 192), (1031, 4096), (2064, 2048)])
@pytest.mark.parametrize("m", [1, 3, 8])
@pytest.mark.parametrize("fmt", ["fp16", "bf16"])
def test_sizes(cuda, n, k, m, fmt):
    from poptransformer_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(n + k + m)
    dt = torch.float16 if fmt == "fp16" else torch.bfloat16
    w, x = (torch.randn((n, k), generator=g, device=cuda) * 0.05).to(dt), torch.randn((m, k), generator=g, device=cuda).to(dt)
    err = torch.zeros(1, dtype=torch.int32, device=cuda)
    out = torch.empty((m, n), dtype=dt, device=cuda)
    ops.gemm(x, ops.GemmWeight(ops.W_FP16 if fmt == "fp16" else ops.W_BF16, w), out=out, error_flag=err)
    exp, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # one rounding of the result, and k sums of which each step may lose 2^-23 of what has gathered
    bound = exp.abs() * 2.0 ** (-11 if fmt == "fp16" else -8) + size * k * 2.0 ** -23 + 1e-6
    assert bool(((out.double() - exp).abs() <= bound).all()) and int(err.item()) == 0


@pytest.mark.parametrize("epilogue", ["residual", "bias", "bias_residual", "bias_gelu", "relu2", "swiglu"])
@pytest.mark.parametrize("n,k", [(768, 768), (768, 3072), (80, 128), (1000, 64)])
def test_fp16_epilogues(cuda, n, k, epilogue):
    """As many roundings as the same steps in fp16; the residual is the output itself, as the decoders have it."""
    from poptransformer_b200 import ops
    if epilogue == "swiglu" and n % 16:
        pytest.skip("gates and ups come in blocks of eight")
    g = torch.Generator(device=cuda).manual_seed(n + k)
    m = 5
    w, x = (torch.randn((n, k), generator=g, device=cuda) * 0.05).half(), torch.randn((m, k), generator=g, device=cuda).half()
    bias, res = torch.randn(n, generator=g, device=cuda).half(), torch.randn((m, n), generator=g, device=cuda).half()
    y = (x.double() @ w.double().T)
    b = bias.double()
    exp = {"residual": res.double() + y, "bias": y + b, "bias_residual": res.double() + y + b, "bias_gelu": torch.nn.functional.gelu(y + b), "relu2": torch.relu(y) ** 2,
           "swiglu": None}[epilogue]
    if epilogue == "swiglu":
        y = y.view(m, -1, 2, 8)
        exp = (torch.nn.functional.silu(y[:, :, 0]) * y[:, :, 1]).reshape(m, -1)
    out = res.clone() if "residual" in epilogue else torch.empty((m, n // 2 if epilogue == "swiglu" else n), dtype=torch.float16, device=cuda)
    ops.gemm(x, ops.GemmWeight(ops.W_FP16, w), out=out, epilogue=getattr(ops, "EPI_" + epilogue.upper()), bias=bias if "bias" in epilogue else None,
             residual=out if "residual" in epilogue else None)
    # three or four roundings of values of the size of the result and of the sums that went into it
    bound = 4 * 2.0 ** -11 * (exp.abs() + 4) * (1 + exp.abs().sqrt())
    assert bool(((out.double() - exp).abs() <= bound).all())


@pytest.mark.parametrize("epilogue", ["store", "residual", "swiglu"])
@pytest.mark.parametrize("n,k", [(768, 768), (768, 3072)])
@pytest.mark.parametrize("m", [1, 8, 9])
def test_fp16_scales(cuda, n, k, m, epilogue):
    """Scales of weights and activations multiply the sums whatever the number of rows (eight is the last that the kernel for few rows takes)."""
    from poptransformer_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(n + k + m)
    w, x = torch.randn((n, k), generator=g, device=cuda).half(), torch.randn((m, k), generator=g, device=cuda).half()
    res = torch.randn((m, n), generator=g, device=cuda).half()
    y = x.double() @ w.double().T * (0.25 * 0.1875)
    exp = res.double() + y if epilogue == "residual" else y
    if epilogue == "swiglu":
        y = y.view(m, -1, 2, 8)
        exp = (torch.nn.functional.silu(y[:, :, 0]) * y[:, :, 1]).reshape(m, -1)
    out = torch.empty_like(exp, dtype=torch.float16)
    ops.gemm(x, ops.GemmWeight(ops.W_FP16, w, w_scale=0.1875), out=out, x_scale=0.25, epilogue=getattr(ops, "EPI_" + epilogue.upper()), residual=res if epilogue == "residual" else None)
    # as in test_fp16_epilogues: three or four roundings of values of the size of the result and of the sums (below eight) that went into it
    assert bool(((out.double() - exp).abs() <= 4 * 2.0 ** -11 * (exp.abs() + 8) * (1 + exp.abs().sqrt())).all())


@pytest.mark.parametrize("rows", [1, 7, 16, 32, 40, 300])
@pytest.mark.parametrize("d,f", [(256, 512), (2048, 8192), (128, 136)])
def test_products_that_share_a_launch(cuda, rows, d, f):
    """Parts give the bits of products of their own, and the gated residual those of the launches it stands for."""
    from poptransformer_b200 import ops
    L, P, S = ops._lib.lib(), ops._ptr, ops._stream
    g = torch.Generator(device=cuda).manual_seed(rows + d)
    w = [(torch.randn((n, d), generator=g, device=cuda) * 0.05).half() for n in (d, d, f)]
    x = torch.randn((3, rows, d), generator=g, device=cuda).half()
    outs = [torch.full((rows, n.shape[0]), 7, dtype=torch.float16, device=cuda) for n in w]
    epi = [ops.EPI_STORE, ops.EPI_RELU2, ops.EPI_RELU2]
    ops.gemm(x.view(-1, d), ops.GemmWeight(ops.W_FP16, torch.cat(w)), parts=list(zip(outs, epi)))
    for i in range(3):
        exp = x[i].double() @ w[i].double().T
        exp = exp if i == 0 else torch.relu(exp) ** 2
        # the rounding of the sum (and of its square), and k sums of which each step may lose 2^-23 of what has gathered
        size = x[i].double().abs() @ w[i].double().abs().T
        assert bool(((outs[i].double() - exp).abs() <= exp.abs() * 2.0 ** -9 + size * d * 2.0 ** -22 * (1 + 2 * exp.sqrt().nan_to_num()) + 1e-6).all())
    gw = ops.GemmWeight(ops.W_FP16, w[0])
    gate, res = torch.randn((rows, d), generator=g, device=cuda).half(), torch.randn((rows, d), generator=g, device=cuda).half()
    for halve in (0, 1):
        want, got = res.clone(), res.clone()
        y = ops.gemm(x[0], gw, ksplit=1)
        ops.check(L.pt_rwkv_ffn_out(P(want), P(gate), P(y), halve, want.numel(), S()), "out")
        ops.gemm(x[0], gw, out=got, epilogue=ops.EPI_GATED_RESIDUAL, residual=got, gate=gate, halve=halve, ksplit=1)
        assert torch.equal(got, want)
        ops.gemm(x[0], gw, out=got.copy_(res), epilogue=ops.EPI_GATED_RESIDUAL, residual=got, gate=gate, halve=halve)
        assert float((got.double() - want.double()).abs().max()) <= 2.0 ** -7      # another order of the sums: a rounding or two of values below four
