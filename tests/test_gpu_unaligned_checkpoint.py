"""Checkpoints whose tensors are views into one buffer, off 16-byte boundaries: what they give as tensors of their own."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _views(sd, cuda, keep):
    """The tensors in one device buffer each, two bytes off; those whose key contains one of `keep` stay as they are."""
    out = {}
    for k, v in sd.items():
        v = v.to(cuda) if torch.is_tensor(v) else v
        if torch.is_tensor(v) and v.dim() and v.element_size() <= 2 and not any(x in k for x in keep):
            off = 2 // v.element_size()
            buf = torch.empty(v.numel() + off, dtype=v.dtype, device=cuda)
            view = buf[off:].view(v.shape)
            view.copy_(v)
            assert view.data_ptr() % 16 == 2
            v = view
        out[k] = v
    return out


@pytest.mark.parametrize("family", ["rwkv", "gpt2", "llama fp16", "llama int4", "chatglm2"])
def test_unaligned_checkpoint(cuda, family):
    from poptransformer_b200 import chatglm2, gpt2, llama, rwkv, synth
    L, G, R = dict(n_layer=2, d_model=256, n_head=2, ffn=512, vocab=500), dict(n_layer=2, d_model=256, n_head=4, vocab=500, n_positions=32), dict(n_layer=2, d_model=256, ffn=512, vocab=500)
    C = dict(n_layer=2, d_model=512, n_head=4, n_group=2, ffn=768, vocab=1000)
    rows, sd, make = {
        "rwkv": (3, synth.rwkv_state_dict(**R, seed=1), lambda s: rwkv.RWKVDecoder(rwkv.RWKVConfig(**R, max_len=32), s, 3, device=cuda)),
        "gpt2": (3, synth.gpt2_state_dict(**G, seed=1), lambda s: gpt2.GPT2Decoder(gpt2.GPT2Config(**G, max_len=32), s, 3, device=cuda)),
        "llama fp16": (4, synth.llama_state_dict(**L, seed=1), lambda s: llama.LlamaDecoder(llama.LlamaConfig(**L, max_len=32), s, 4, device=cuda)),
        "llama int4": (12, synth.llama_state_dict(**L, seed=1, int4_group=128), lambda s: llama.LlamaDecoder(llama.LlamaConfig(**L, max_len=32, int4_group=128), s, 12, device=cuda)),
        "chatglm2": (3, synth.chatglm2_state_dict(**C, seed=1), lambda s: chatglm2.ChatGLM2Decoder(chatglm2.ChatGLM2Config(**C, max_len=32), s, 3, device=cuda)),
    }[family]
    logits = []
    for s in (sd, _views(sd, cuda, keep=("emb", "wte", "wpe"))):       # (embedding rows are read 16 bytes at a time)
        dec = make(s)
        dec.reset(synth.prompt_ids(rows, 5, 32, dec.cfg.vocab, dec.pad_id, seed=2))
        for _ in range(4):
            dec.step()
        logits.append(dec.logits.clone())
    a, b = (x.double() for x in logits)       # (norms off the boundary add up in another order: roundings to fp16 that fall the other way)
    assert float((a - b).norm() / a.norm()) < 1e-2
