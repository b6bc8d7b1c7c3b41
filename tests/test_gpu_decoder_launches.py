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
