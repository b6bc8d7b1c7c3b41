"""What the decoders hand to the linears and the attention they launch."""
import pytest
import torch

pytestmark = pytest.mark.gpu

LLAMA = dict(n_layer=2, d_model=256, n_head=2, ffn=512, vocab=500)


def _llama(cuda, batch, group, **kw):
    from poptransformer_b200 import llama, synth
    return llama.LlamaDecoder(llama.LlamaConfig(**LLAMA, max_len=64, int4_group=group), synth.llama_state_dict(**LLAMA, seed=3, device="cpu", int4_group=group), batch, device=cuda, **kw)


@pytest.mark.parametrize("batch", [1, 4, 12])
@pytest.mark.parametrize("group", [0, 128])
def test_linears_alone(cuda, batch, group):
    """enqueue_linears_only() runs the four products of every block, whatever kernel serves them."""
    from poptransformer_b200 import synth
    dec = _llama(cuda, batch, group, persistent=None if batch > 2 else False)
    dec.x.normal_(0, 0.5)
    dec.attn.normal_(0, 0.5)
    dec.h.normal_(0, 0.5)         # (the GEMM route leaves the norms out)
    dec.enqueue_linears_only()
    sd = synth.llama_state_dict(**LLAMA, seed=3, device="cpu", int4_group=group)
    key = f"model.layers.{LLAMA['n_layer'] - 1}.mlp.down_proj.weight"
    w = sd[key]
    if group:       # byte j: k = 2 j in the high nibble, 2 j + 1 in the low, two's complement
        w = torch.stack([w >> 4, (w << 4) >> 4], 2).reshape(w.shape[0], -1).double() * sd[key + "_scale"].reshape(w.shape[0], -1).double().repeat_interleave(group, 1)
    want = dec.act.double() @ w.to(cuda).double().T
    assert float((dec.part.double() - want).norm() / want.norm()) < 2e-3      # fp16 rounding of the result and, on the GEMM, of nibble times scale


class _Calls:
    """Records what is passed to ops.gemm, ops.linear, ops.linear_args and ops.attn_args."""

    def __init__(self, monkeypatch):
        from poptransformer_b200 import ops
        self.gemm, self.linear, self.attn = [], [], []
        gemm, linear_args, attn_args = ops.gemm, ops.linear_args, ops.attn_args

        def seen_gemm(*a, **kw):
            self.gemm.append(kw)
            return gemm(*a, **kw)

        def seen_linear(*a, **kw):
            self.linear.append(kw)
            return linear_args(*a, **kw)

        def seen_attn(*a, **kw):
            self.attn.append(kw)
            return attn_args(*a, **kw)

        monkeypatch.setattr(ops, "gemm", seen_gemm)
        monkeypatch.setattr(ops, "linear_args", seen_linear)
        monkeypatch.setattr(ops, "attn_args", seen_attn)


def _decoders(cuda, only=None, **kw):
    """name -> a decoder with its linears on the GEMM (kw: constructor arguments that all take, pdl / pdl_linear / pdl_attn as each has them)."""
    from poptransformer_b200 import chatglm2, gpt2, rwkv, synth
    off = kw.pop("off", False)
    both = dict(pdl_linear=0, pdl_attn=0) if off else {}
    g2 = dict(n_layer=2, d_model=256, n_head=4, vocab=500, n_positions=64)
    glm = dict(n_layer=2, d_model=512, n_head=4, n_group=2, ffn=768, vocab=1000)
    rw = dict(n_layer=2, d_model=256, ffn=512, vocab=500)
    make = {
        "llama fp16": lambda: _llama(cuda, 4, 0, **(dict(pdl=False) if off else {})),
        "llama int4": lambda: _llama(cuda, 12, 128, prefill=True, **(dict(pdl=False) if off else {})),
        "gpt2": lambda: gpt2.GPT2Decoder(gpt2.GPT2Config(**g2, max_len=64), synth.gpt2_state_dict(**g2, seed=1), 3, device=cuda, **both),
        "chatglm2 fp16": lambda: chatglm2.ChatGLM2Decoder(chatglm2.ChatGLM2Config(**glm, max_len=64), synth.chatglm2_state_dict(**glm, seed=1), 3, device=cuda, **both),
        "chatglm2 fp8": lambda: chatglm2.ChatGLM2Decoder(chatglm2.ChatGLM2Config(**glm, max_len=64, precision="fp8"), synth.chatglm2_state_dict(**glm, seed=1, precision="fp8"), 8,
                                                         device=cuda, **both),
        "rwkv": lambda: rwkv.RWKVDecoder(rwkv.RWKVConfig(**rw, max_len=64), synth.rwkv_state_dict(**rw, seed=1), 3, device=cuda, **({"pdl_linear": 0} if off else {})),
    }
    return {k: f() for k, f in make.items()}


def _ids(dec):
    from poptransformer_b200 import synth
    return synth.prompt_ids(dec.batch, 6, dec.cfg.max_len, dec.cfg.vocab, dec.pad_id, seed=5)


def test_products_can_report(cuda, monkeypatch):
    """A product whose waits run out leaves its output as it was: the decoder's error flag is the only sign of it."""
    for name, dec in _decoders(cuda).items():
        seen = _Calls(monkeypatch)
        dec.reset(_ids(dec))
        if name == "llama int4":
            dec.prefill()
        dec.step()
        assert seen.gemm and all(kw.get("error_flag") is dec.error_flag for kw in seen.gemm), name
        monkeypatch.undo()


def test_early_starts_can_be_switched_off(cuda, monkeypatch):
    outs = []
    for off in (False, True):
        for name, dec in _decoders(cuda, off=off).items():
            seen = _Calls(monkeypatch)
            dec.reset(_ids(dec))
            if name == "llama int4":
                dec.prefill()
            dec.step()
            early = [int(kw.get("pdl", 0)) for kw in seen.gemm + seen.linear + seen.attn]
            assert seen.gemm and not any(early) if off else any(early), (name, off)
            if not off and name != "rwkv":       # (products on side streams have no launch of their stream in front)
                assert all(early), name
            outs.append(dec.logits.clone())
            monkeypatch.undo()
    n = len(outs) // 2
    assert all(torch.equal(a, b) for a, b in zip(outs[:n], outs[n:]))


def test_no_workspace_that_nothing_uses(cuda):
    """Only the skinny-matmul kernels sum k-slices in a workspace (16 slices x rows x outputs in fp32)."""
    for name, dec in _decoders(cuda).items():
        assert dec.lin_ws is None and not any(w is not None for w in getattr(dec, "side_ws", [])), name
    few = _llama(cuda, 1, 0)                                      # fp16 blocks on the GEMM, the output layer on the skinny-matmul kernel
    assert few.lin_ws is not None and few.lin_ws.numel() < 16 * LLAMA["vocab"] * 4 + (1 << 20)
