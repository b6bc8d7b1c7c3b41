"""A ragged number of rows or of outputs takes a product no longer than the whole one above it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _us(fns):
    for f in fns[:2]:
        f()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for f in fns:
            f()
    best = 1e9
    for _ in range(8):
        e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        e0.record()
        g.replay()
        e1.record()
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1) * 1e3 / len(fns))
    return best


def _product(cuda, fmt, n, k, m, copies=12):
    from poptransformer_b200 import ops
    if fmt == "int4":
        ws = [ops.GemmWeight(ops.W_INT4, torch.randint(-128, 127, (n, k // 2), dtype=torch.int8, device=cuda), torch.rand((n, k // 128), device=cuda).half() * 0.01, group=128)
              for _ in range(copies)]
    else:
        ws = [ops.GemmWeight(ops.W_FP8, torch.randint(0, 100, (n, k), dtype=torch.uint8, device=cuda), w_scale=0.01) for _ in range(copies)]
    x = torch.randn((m, k), device=cuda).half() if fmt == "int4" else torch.randint(0, 100, (m, k), dtype=torch.uint8, device=cuda)
    out = torch.empty((m, n), dtype=torch.float16, device=cuda)
    return _us([lambda w=w: ops.gemm(x, w, out=out) for w in ws])


# (format, n, k, m, then the whole n and m): rows that fill a step of 16 in part; a last tile that is half empty
@pytest.mark.parametrize("fmt,n,k,m,n_whole,m_whole", [("fp8", 2048, 128, 12, 2048, 16), ("int4", 2048, 128, 12, 2048, 16), ("fp8", 10304, 2048, 256, 10368, 256)])
def test_ragged_sizes_take_no_longer(cuda, fmt, n, k, m, n_whole, m_whole):
    ragged, whole = (min(_product(cuda, fmt, *size) for _ in range(3)) for size in ((n, k, m), (n_whole, k, m_whole)))
    assert ragged <= 1.15 * whole, (ragged, whole)      # (1.3 to 1.5 when such steps and tiles left element by element)


@pytest.mark.parametrize("epilogue", ["store", "bias", "residual", "bias_residual", "gelu", "relu2", "swiglu"])
@pytest.mark.parametrize("n", [16, 48, 144, 1040, 1003])        # a quarter of a tile or part of one in use, whole quarters empty, an odd row length
@pytest.mark.parametrize("m", [1, 7, 16, 23])
def test_ragged_epilogues(cuda, epilogue, n, m):
    """Every fp16 epilogue against the stored sums, in rows of their own and in rows off 4-byte boundaries."""
    from poptransformer_b200 import ops
    if epilogue == "swiglu" and n % 16:
        pytest.skip("features in blocks of eight")
    k = 64
    w, x = torch.randn((n, k), device=cuda).half() * 0.2, torch.randn((m, k), device=cuda).half()
    res, bias = torch.randn((m, n), device=cuda).half(), torch.randn((n,), device=cuda).half()
    gw = ops.GemmWeight(ops.W_FP16, w)
    y = ops.gemm(x, gw, ksplit=1)
    assert float((y.double() - x.double() @ w.double().T).abs().max()) < 2e-2
    want, kw = {
        "store": lambda: (y, {}), "bias": lambda: (y + bias, dict(epilogue=ops.EPI_BIAS, bias=bias)), "residual": lambda: (res + y, dict(epilogue=ops.EPI_RESIDUAL, residual=res)),
        "bias_residual": lambda: (res + (y + bias), dict(epilogue=ops.EPI_BIAS_RESIDUAL, bias=bias, residual=res)),
        "gelu": lambda: (None, dict(epilogue=ops.EPI_BIAS_GELU, bias=bias)), "relu2": lambda: (y.clamp_min(0) * y.clamp_min(0), dict(epilogue=ops.EPI_RELU2)),
        "swiglu": lambda: (None, dict(epilogue=ops.EPI_SWIGLU)),
    }[epilogue]()
    cols = n // 2 if epilogue == "swiglu" else n
    if epilogue == "gelu":
        want = torch.nn.functional.gelu((y + bias).float()).half()
    if epilogue == "swiglu":
        v = y.view(m, n // 16, 2, 8)
        want = (v[:, :, 1] * torch.nn.functional.silu(v[:, :, 0].float()).half()).reshape(m, cols)
    for ld, off in ((cols, 0), (cols + 3, 1)):
        buf = torch.full((m * ld + 8,), 7.0, dtype=torch.float16, device=cuda)
        out = buf[off:off + m * ld]
        ops.gemm(x, gw, out=out, out_ld=ld, ksplit=1, **kw)
        got = out.view(m, ld)
        if epilogue in ("gelu", "swiglu"):               # (another exponential: one more rounding to fp16)
            assert torch.allclose(got[:, :cols].float(), want.float(), rtol=2.0 ** -9, atol=2.0 ** -16)
        else:
            assert torch.equal(got[:, :cols], want)
        assert bool((got[:, cols:] == 7).all()) and bool((buf[:off] == 7).all()) and bool((buf[off + m * ld:] == 7).all())
