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


@pytest.mark.parametrize("family", ["gpt2", "chatglm2", "rwkv"])
def test_capture_leaves_the_stop_state(cuda, family):
    """A step captured just before a row's eos id comes: the row ends with the replayed iteration, not with the one that capture() runs."""
    from poptransformer_b200 import chatglm2, gpt2, rwkv, synth
    max_len, at = 32, 9
    dims = dict(n_layer=2, d_model=256, vocab=500)
    if family == "gpt2":
        dims.update(n_head=4, n_positions=max_len)
        sd, cfg, decoder = synth.gpt2_state_dict(**dims, seed=1), gpt2.GPT2Config(**dims, max_len=max_len), gpt2.GPT2Decoder
    elif family == "chatglm2":
        dims.update(n_head=4, n_group=2, ffn=384)
        sd, cfg, decoder = synth.chatglm2_state_dict(**dims, seed=1), chatglm2.ChatGLM2Config(**dims, max_len=max_len), chatglm2.ChatGLM2Decoder
    else:
        dims.update(ffn=512)
        sd, cfg, decoder = synth.rwkv_state_dict(**dims, seed=1), rwkv.RWKVConfig(**dims, max_len=max_len), rwkv.RWKVDecoder
    ids = synth.prompt_ids(1, 20, max_len, 400, dims["vocab"] - 1, seed=2)
    ids[0, at] = 450                    # the end, at a place that only the test knows
    make = lambda: decoder(cfg, sd, 1, device=cuda, pad_id=dims["vocab"] - 1, eos_id=450, early_stop=True)      # noqa: E731
    want = make().run(ids, max_loop=20)
    dec = make()
    dec.reset(ids)
    for _ in range(at - 1):
        dec.step()
    dec.capture()
    assert dec.step_t.item() == at - 1 and not dec.stop_mask.any() and not dec.done_flag.any()
    for _ in range(at - 1, 20):
        dec.step()
    assert (dec.ids.cpu().numpy() == want["Loop:0"]).all() and dec.step_t.item() == want["Loop:1"].item() == at + 1
