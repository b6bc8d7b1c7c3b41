"""The fused element-wise kernels of RWKV give the bits of the launches they stand for."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,dim", [(1, 8), (1, 2048), (32, 2048), (5, 8184)])
def test_fused_launches_match(cuda, rows, dim):
    from poptransformer_b200 import ops
    L, P, S = ops._lib.lib(), ops._ptr, ops._stream
    g = torch.Generator(device=cuda).manual_seed(rows + dim)
    rnd = lambda *s: torch.randn(s, device=cuda, generator=g).half()
    x, gamma, beta, state = rnd(rows, dim), rnd(dim), rnd(dim), rnd(rows, dim)
    mixes = [torch.rand(dim, device=cuda, generator=g).half() for _ in range(3)]
    for n in (1, 2, 3):
        w = [P(m) for m in mixes[:n]] + [None] * (3 - n)
        t, s1, s2 = torch.empty_like(x), state.clone(), state.clone()
        a, b = ([torch.full_like(x, 7) for _ in range(n)] for _ in range(2))
        ops.check(L.pt_norm_ce(P(x), P(gamma), P(beta), rows, dim, 1e-5, P(t), S()), "norm")
        ops.check(L.pt_rwkv_mix(P(t), P(s1), *w, *[P(o) for o in a], *[None] * (3 - n), rows, dim, S()), "mix")
        ops.check(L.pt_norm_ce_mix(P(x), P(gamma), P(beta), rows, dim, 1e-5, P(s2), *w, *[P(o) for o in b], *[None] * (3 - n), S()), "norm mix")
        assert torch.equal(s1, s2) and all(torch.equal(p, q) for p, q in zip(a, b))
    r, v = rnd(rows, dim), rnd(rows, dim)
    for halve in (0, 1):
        gate, want, got = torch.empty_like(x), torch.empty_like(x), x.clone()
        ops.check(L.pt_rwkv_act(0, P(r), P(v), P(gate), r.numel(), S()), "act")
        ops.check(L.pt_add_f16(P(x), P(gate), x.numel(), P(want), S()), "add")
        if halve:
            ops.check(L.pt_rwkv_act(2, P(want), None, P(want), x.numel(), S()), "act")
        ops.check(L.pt_rwkv_ffn_out(P(got), P(r), P(v), halve, x.numel(), S()), "out")
        assert torch.equal(got, want)
    tf, td = torch.randn(dim, device=cuda, generator=g), torch.randn(dim, device=cuda, generator=g)
    st = [[torch.rand((rows, dim), device=cuda, generator=g), torch.rand((rows, dim), device=cuda, generator=g) + 1, torch.randn((rows, dim), device=cuda, generator=g)]]
    st.append([t.clone() for t in st[0]])
    want, got = torch.empty_like(x), torch.empty_like(x)
    ops.check(L.pt_wkv(P(x), P(v), P(tf), P(td), *[P(t) for t in st[0]], rows, dim, P(want), S()), "wkv")
    ops.check(L.pt_rwkv_act(0, P(r), P(want), P(want), x.numel(), S()), "act")
    ops.check(L.pt_wkv_gated(P(x), P(v), P(r), P(tf), P(td), *[P(t) for t in st[1]], rows, dim, P(got), S()), "wkv gated")
    assert torch.equal(got, want) and all(torch.equal(p, q) for p, q in zip(*st))


@pytest.mark.parametrize("rows", [1, 32, 70])
def test_squared_relu_epilogue(cuda, rows):
    from poptransformer_b200 import ops
    w, x = torch.randn((1000, 512), device=cuda).half() * 0.05, torch.randn((rows, 512), device=cuda).half()
    gw = ops.GemmWeight(ops.W_FP16, w)
    for ksplit in (0, 1):
        y = ops.gemm(x, gw, ksplit=ksplit).clamp_min(0)
        assert torch.equal(ops.gemm(x, gw, epilogue=ops.EPI_RELU2, ksplit=ksplit), y * y)


def test_captured_step_keeps_the_state(cuda):
    """capture() leaves ids, step and states as they were, and replayed steps give what launched ones give."""
    from poptransformer_b200 import rwkv, synth
    dims = dict(n_layer=2, d_model=256, ffn=512, vocab=500)
    sd = synth.rwkv_state_dict(**dims, seed=1, device="cpu")
    ids = synth.prompt_ids(3, 6, 16, dims["vocab"], dims["vocab"] - 1, seed=2)
    dec = rwkv.RWKVDecoder(rwkv.RWKVConfig(**dims, max_len=16), sd, 3, device=cuda)
    want = dec.run(ids, max_loop=10)
    dec.reset(ids)
    for _ in range(4):
        dec.step()
    dec.capture()
    for _ in range(6):
        dec.step()
    assert (dec.ids.cpu().numpy() == want["Loop:0"]).all() and dec.step_t.item() == want["Loop:1"].item()
