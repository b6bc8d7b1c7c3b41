"""ChatGLM2's replayed steps give what launched ones give, wherever in a generation they were captured."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,rows", [("fp16", 3), ("fp8", 2), ("fp8", 8)])     # fp16 on the GEMM, FP8 on the skinny-matmul kernels and on the GEMM
def test_chatglm2_replays(cuda, precision, rows):
    import torch
    from poptransformer_b200 import chatglm2, synth
    dims, max_len = dict(n_layer=2, d_model=512, n_head=4, n_group=2, ffn=768, vocab=1000), 80
    sd = synth.chatglm2_state_dict(**dims, seed=1, device="cpu", precision=precision)
    dec = chatglm2.ChatGLM2Decoder(chatglm2.ChatGLM2Config(**dims, max_len=max_len, precision=precision), sd, rows, device=cuda)
    ids = synth.prompt_ids(rows, 6, max_len, dims["vocab"], dec.pad_id, seed=2)
    want, logits = dec.run(ids, max_loop=70), dec.logits.clone()
    dec.reset(ids)
    for _ in range(4):
        dec.step()
    dec.capture()
    assert dec.graph is not None and dec.step_t.item() == 4
    n = []
    enqueue, dec.enqueue_step = dec.enqueue_step, lambda: n.append(enqueue())
    for _ in range(66):          # across the edge of a cache page
        dec.step()
    assert not n                 # replayed
    assert (dec.ids.cpu().numpy() == want["Loop:0"]).all() and dec.step_t.item() == want["Loop:1"].item() and torch.equal(dec.logits, logits)
    assert (dec.run(ids, max_loop=70)["Loop:0"] == want["Loop:0"]).all() and not n     # from the start with the same graph
