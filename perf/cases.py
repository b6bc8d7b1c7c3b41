"""The work that a user of this framework has it do, as cases that can be timed and compared.

A case is one call, or a short run of calls, through a decoder's public methods: a decode step of a batch at some context, a prompt
and the first token after it, a few iterations of the loop from its start, or a batch of requests of unequal lengths that is served
to its end.  Weights, prompts and caches are random, of the shapes and value ranges of the architectures in MODELS.

`exact` computes the same in 64 bits from the same weights with torch alone: what the models define as rounded (INT4 and E4M3
values, the E4M3 cast of the activations, the fp16 sine and cosine tables) is rounded there too, nothing else is.
"""
import math

import numpy as np
import torch

MODELS = {
    "gpt2-small": dict(family="gpt2", layers=12, d=768, heads=12, vocab=50257),
    "gpt2-xl": dict(family="gpt2", layers=48, d=1600, heads=25, vocab=50257),
    "llama-7b": dict(family="llama", layers=32, d=4096, heads=32, ffn=11008, vocab=32000),
    "llama-2k": dict(family="llama", layers=16, d=2048, heads=16, ffn=8192, vocab=32000),
    "chatglm2-6b": dict(family="glm", layers=28, d=4096, heads=32, groups=2, ffn=13696, vocab=65024),
    "rwkv4-1b5": dict(family="rwkv", layers=24, d=2048, ffn=8192, vocab=50277),
    "sabisun-2k": dict(family="sabisun", layers=16, d=2048, ffn=8192, heads=16, kv_heads=4, ssm_heads=64, window=1024, keep_first=64, streams=2, vocab=32000),
    "sabisun-4k": dict(family="sabisun", layers=16, d=4096, ffn=14336, heads=32, kv_heads=8, ssm_heads=128, window=1024, keep_first=64, streams=4, vocab=32000),
}
PAGE = 64            # positions of a cache page, as the decoders have it by default
POSITIONS = 1024     # GPT-2's learned positions


def listed():
    return [
        # The smallest call: one sequence of a small model, where launches and latency are what a token costs.
        dict(name="gpt2-small step", model="gpt2-small", mode="decode", weights="fp16", layers=12, rows=1, context=159),
        # The largest GPT-2 for sixteen sequences (four prompts with four hypotheses each have as many rows); 25 heads, width 1600.
        dict(name="gpt2-xl step 16 rows", model="gpt2-xl", mode="decode", weights="fp16", layers=48, rows=16, context=255),
        # Chat with one user on a 7B model with INT4 weights: the headline workload.
        dict(name="llama-7b step", model="llama-7b", mode="decode", weights="int4", group=128, layers=32, rows=1, context=511),
        # The same model serving a batch ...
        dict(name="llama-7b step 16 rows", model="llama-7b", mode="decode", weights="int4", group=128, layers=32, rows=16, context=511),
        # ... and a larger one at a shorter context.
        dict(name="llama-7b step 32 rows", model="llama-7b", mode="decode", weights="int4", group=128, layers=32, rows=32, context=255),
        # Time to the first token: a prompt in one pass, then the step that reads its last token.
        dict(name="llama-7b prompt", model="llama-7b", mode="prompt", weights="int4", group=128, layers=32, rows=1, context=511),
        # fp16 weights (the reference's default precision), multi-query attention, a long context, a small batch.
        dict(name="chatglm2 step 8 rows", model="chatglm2-6b", mode="decode", weights="fp16", layers=28, rows=8, context=1151),
        # FP8 through the operator surface: the casts and products of the matrices of four blocks and the output layer.  (Not as whole
        # steps: casts whose input lies between two E4M3 values make two right implementations drift apart by several per cent within
        # one block.)
        dict(name="chatglm2 fp8 products 8 rows", model="chatglm2-6b", mode="products", weights="fp8", layers=4, rows=8, context=0),
        # A recurrent model takes a prompt token by token: eight iterations of the loop for 32 sequences.
        dict(name="rwkv loop 32 rows", model="rwkv4-1b5", mode="loop", weights="fp16", layers=24, rows=32, context=8),
        # Hybrid decoder (attention and state-space layers), a step of a small batch behind long prompts.
        dict(name="sabisun-2k step 8 rows", model="sabisun-2k", mode="decode", weights="bf16", layers=16, rows=8, context=2047),
        # A long prompt of one sequence, logits of its last token.
        dict(name="sabisun-2k prompt", model="sabisun-2k", mode="serve", weights="bf16", layers=16, rows=1, context=2048, tokens=0),
        # Requests of unequal lengths: all prompts as one batch, then six more tokens each, then they end.
        dict(name="sabisun-2k requests", model="sabisun-2k", mode="serve", weights="bf16", layers=16, rows=7, context=600, tokens=6),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    model = rng.choice(["gpt2-small", "gpt2-xl", "llama-7b", "llama-7b", "llama-7b", "llama-2k", "chatglm2-6b", "chatglm2-6b", "rwkv4-1b5", "sabisun-2k", "sabisun-2k", "sabisun-4k"])
    m = MODELS[model]
    c = dict(model=model, mode="decode", weights="fp16", layers=rng.randint(1, min(12, m["layers"])), rows=log(1, 32), context=log(1, 1000))
    if m["family"] == "llama":
        c["weights"] = rng.choice(["int4", "int4", "fp16"])
        if c["weights"] == "int4":
            c["group"] = rng.choice([128, 128, 256])
            c["mode"] = rng.choice(["decode", "decode", "prompt"])
        if c["mode"] == "prompt":
            c["rows"], c["context"] = rng.randint(1, 3), log(8, 1000)
    elif m["family"] == "glm":
        if rng.random() < 0.5:
            c["weights"], c["mode"], c["layers"], c["rows"], c["context"] = "fp8", "products", rng.randint(1, 4), log(1, 200), 0
    elif m["family"] == "rwkv":
        c["mode"], c["context"] = "loop", rng.randint(1, 8)
    elif m["family"] == "sabisun":
        c["weights"], c["mode"] = "bf16", rng.choice(["decode", "serve"])
        c["layers"] = rng.randint(4, 12)
        if c["mode"] == "serve":
            c["rows"], c["tokens"] = log(1, 8), rng.choice([0, rng.randint(1, 8)])
    return c


# ------------------------------------------------------------------------------------------ weights and inputs
def _gen(seed, part=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + part)


def _normal(shape, g, std=0.02, mean=0.0, dtype=torch.float16):
    return torch.empty(shape, dtype=torch.float32, device="cuda").normal_(mean, std, generator=g).to(dtype)


def _int4(n, k, group, g):
    """Signed nibbles of a normal distribution, even k in the high half of a byte, and a scale per row and group."""
    q = torch.empty((n, k), dtype=torch.float32, device="cuda").normal_(0.0, 2.6, generator=g).round_().clamp_(-7, 7).to(torch.int8)
    w = ((q[:, 0::2] << 4) | (q[:, 1::2] & 15)).contiguous()
    return w, (torch.rand((n, k // group), generator=g, device="cuda") * 0.003 + 0.006).to(torch.float16)


def _weights(case, seed):
    m, L, g = MODELS[case["model"]], case["layers"], _gen(seed)
    return {"gpt2": _gpt2_weights, "llama": _llama_weights, "glm": _glm_weights, "rwkv": _rwkv_weights, "sabisun": _sabisun_weights}[m["family"]](case, m, L, g)


def _norms(sd, g, d, *keys, bias=False, dtype=torch.float16):
    for k in keys:
        sd[k + ".weight"] = _normal((d,), g, 0.02, 1.0, dtype)
        if bias:
            sd[k + ".bias"] = _normal((d,), g, 0.02, 0.0, dtype)


def _gpt2_weights(case, m, L, g):
    d = m["d"]
    sd = {"transformer.wte.weight": _normal((m["vocab"], d), g), "transformer.wpe.weight": _normal((POSITIONS, d), g)}
    for i in range(L):
        p = f"transformer.h.{i}."
        _norms(sd, g, d, p + "ln_1", p + "ln_2", bias=True)
        for key, o, k in (("attn.c_attn", 3 * d, d), ("attn.c_proj", d, d), ("mlp.c_fc", 4 * d, d), ("mlp.c_proj", d, 4 * d)):
            sd[p + key + ".weight"], sd[p + key + ".bias"] = _normal((o, k), g), _normal((o,), g)
        for q in ("weight", "bias"):       # the checkpoints come with the query scaled
            sd[p + "attn.c_attn." + q][:d] *= (d // m["heads"]) ** -0.5
    _norms(sd, g, d, "transformer.ln_f", bias=True)
    return sd


def _llama_weights(case, m, L, g):
    d, f = m["d"], m["ffn"]
    sd = {"model.embed_tokens.weight": _normal((m["vocab"], d), g), "lm_head.weight": _normal((m["vocab"], d), g)}
    for i in range(L):
        p = f"model.layers.{i}."
        _norms(sd, g, d, p + "input_layernorm", p + "post_attention_layernorm")
        for key, o, k in [(f"self_attn.{n}_proj", d, d) for n in "qkvo"] + [("mlp.gate_proj", f, d), ("mlp.up_proj", f, d), ("mlp.down_proj", d, f)]:
            key = p + key + ".weight"
            if case["weights"] == "int4":
                sd[key], sd[key + "_scale"] = _int4(o, k, case["group"], g)
            else:
                sd[key] = _normal((o, k), g)
    _norms(sd, g, d, "model.norm")
    return sd


def _glm_weights(case, m, L, g):
    d, f, kv = m["d"], m["ffn"], 2 * m["groups"] * (m["d"] // m["heads"])
    sd = {"transformer.embedding.word_embeddings.weight": _normal((m["vocab"], d), g)}
    for i in range(L):
        p = f"transformer.encoder.layers.{i}."
        _norms(sd, g, d, p + "input_layernorm", p + "post_attention_layernorm")
        for key, o, k in (("self_attention.query", d, d), ("self_attention.key_value", kv, d), ("self_attention.dense", d, d), ("mlp.dense_h_to_4h_1", f, d),
                          ("mlp.dense_h_to_4h_2", f, d), ("mlp.dense_4h_to_h", d, f)):
            sd[p + key + ".weight"] = _normal((o, k), g)
        sd[p + "self_attention.query.bias"], sd[p + "self_attention.key_value.bias"] = _normal((d,), g), _normal((kv,), g)
    _norms(sd, g, d, "transformer.encoder.final_layernorm")
    sd["transformer.output_layer.weight"] = _normal((m["vocab"], d), g)
    return sd


def _products(case, seed):
    """[(weights in E4M3 [n, k], their scale, activations in fp16, the scale they are cast with)] of a model's FP8 linears."""
    m, g = MODELS[case["model"]], _gen(seed)
    d, f, kv = m["d"], m["ffn"], 2 * m["groups"] * (m["d"] // m["heads"])
    block = [(d + kv, d, 1.0, 8.0), (d, d, 0.3, 2.0), (2 * f, d, 1.0, 8.0), (d, f, 0.8, 6.0)]
    out = []
    for n, k, std, reach in block * case["layers"] + [(m["vocab"], d, 1.0, 8.0)]:
        scale = 0.11 / 448.0
        w = (_normal((n, k), g, dtype=torch.float32) / scale).clamp_(-448.0, 448.0).to(torch.float8_e4m3fn).view(torch.uint8)
        out.append((w, scale, _normal((case["rows"], k), g, std), reach / 448.0))
    return out


def _rwkv_weights(case, m, L, g):
    d, f = m["d"], m["ffn"]
    sd = {"rwkv.embeddings.weight": _normal((m["vocab"], d), g, 1.0)}

    def uniform(lo, hi):
        return torch.rand((d,), generator=g, device="cuda") * (hi - lo) + lo

    for i in range(L):
        p = f"rwkv.blocks.{i}."
        a, b, div = p + "attention.", p + "feed_forward.", float(2 ** (i // 6))
        _norms(sd, g, d, *([p + "pre_ln"] if i == 0 else []), p + "ln1", p + "ln2", bias=True)
        sd[a + "time_decay"], sd[a + "time_first"] = uniform(-5.0, -1.0), uniform(-1.0, 1.0)
        for k in (a + "time_mix_key", a + "time_mix_value", a + "time_mix_receptance", b + "time_mix_key", b + "time_mix_receptance"):
            sd[k] = uniform(0.0, 1.0).to(torch.float16).reshape(1, 1, d)
        for k, o, i_, s in ((a + "key", d, d, 1.0), (a + "value", d, d, 1.0), (a + "receptance", d, d, 1.0), (a + "output", d, d, div),
                            (b + "key", f, d, 1.0), (b + "receptance", d, d, 1.0), (b + "value", d, f, div)):
            sd[k + ".weight"] = _normal((o, i_), g, 0.05 / s)
    _norms(sd, g, d, "rwkv.ln_out", bias=True)
    sd["head.weight"] = _normal((m["vocab"], d), g)
    return sd


def _sabisun_config(case):
    """Three state-space layers, then one attention layer, repeated."""
    m = MODELS[case["model"]]
    mamba = {"type": "mamba2", "mixer": {"heads": m["ssm_heads"], "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}}
    attn = {"type": "attention", "mixer": {"heads": m["heads"], "kv_heads": m["kv_heads"], "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                                           "mask": {"size": m["window"], "keep_first": m["keep_first"]}}}
    return {"architecture": "Sabisun", "vocab": m["vocab"], "width": m["d"], "streams": m["streams"], "norm": {"eps": 1e-5}, "residual_mult": 1.0,
            "logit_scale": 1.0, "layers": [dict(attn if i % 4 == 3 else mamba, mlp={"ff": m["ffn"], "kind": "dense"}) for i in range(case["layers"])]}


def _sabisun_weights(case, m, L, g):
    cfg, W, S, sd = _sabisun_config(case), m["d"], m["streams"], {}

    def put(key, shape, std=1.0, mean=0.0):
        sd[key] = _normal(shape, g, std, mean, torch.bfloat16)

    def lin(key, o, k):
        put(key, (o, k), k ** -0.5)

    put("embed", (m["vocab"], W))
    put("final.norm", (W,), 0.02, 1.0)
    for i, lay in enumerate(cfg["layers"]):
        p, x = f"l{i}.", lay["mixer"]
        for q in "12":
            put(p + "norm" + q, (W,), 0.02, 1.0)
            put(p + f"hc{q}.in", (S,), 0.02, 1.0 / S)
            put(p + f"hc{q}.out", (S,), 0.02, 1.0)
            put(p + f"hc{q}.mix", (S, S), 0.02)
            sd[p + f"hc{q}.mix"] += torch.eye(S, device="cuda", dtype=torch.bfloat16)
        if lay["type"] == "attention":
            for n, h in (("q", x["heads"]), ("k", x["kv_heads"]), ("v", x["kv_heads"])):
                lin(p + "mix." + n, h * x["dim"], W)
            put(p + "mix.sink", (x["heads"],))
            lin(p + "mix.o", W, x["heads"] * x["vdim"])
        else:
            inner, ch = x["heads"] * x["vdim"], x["heads"] * x["vdim"] + 2 * x["groups"] * x["state"]
            lin(p + "mix.in", inner + ch + x["heads"], W)
            put(p + "mix.conv", (ch, x["conv"]), 0.5)
            put(p + "mix.conv.b", (ch,), 0.1)
            put(p + "mix.dt_bias", (x["heads"],), 1.0, -3.0)
            put(p + "mix.A_log", (x["heads"],), 1.0, 1.0)
            put(p + "mix.D", (x["heads"],), 0.1, 1.0)
            put(p + "mix.norm", (inner,), 0.02, 1.0)
            lin(p + "mix.o", W, inner)
        lin(p + "mlp.up", m["ffn"], W)
        lin(p + "mlp.down", W, m["ffn"])
    return sd


def _max_len(case):
    """Room behind the context for what a program would generate."""
    return min(-(-(case["context"] + 192) // 64) * 64, POSITIONS if MODELS[case["model"]]["family"] == "gpt2" else 1 << 20)


def _ids(case, seed, n):
    """Prompts of n tokens in a container padded with the last id of the vocabulary."""
    m, r = MODELS[case["model"]], np.random.default_rng([int(seed), 7])
    ids = np.full((case["rows"], _max_len(case)), m["vocab"] - 1, np.int32)
    ids[:, :n] = r.integers(0, m["vocab"] - 1, (case["rows"], n))
    return torch.from_numpy(ids)


def _requests(case, seed):
    """Prompts (one of `context` tokens, the others shorter) and the tokens that follow each of them."""
    m, r = MODELS[case["model"]], np.random.default_rng([int(seed), 9])
    n = case["context"]
    lens = [n] + [max(1, int(n * f)) for f in (0.06, 0.81, 0.35, 0.52, 0.021, 0.97)[:case["rows"] - 1]]
    lens += [max(1, n // 2 + k) for k in range(case["rows"] - len(lens))]
    return [r.integers(0, m["vocab"] - 1, k).astype(np.int32) for k in lens], r.integers(0, m["vocab"] - 1, (case["tokens"], case["rows"])).astype(np.int32)


def _history(case, seed, layer, heads, dim):
    """Keys and values of the positions before the step, [2, rows, heads, context, dim]."""
    return _normal((2, case["rows"], heads, case["context"], dim), _gen(seed, 1 + layer), 0.5)


def _fill(cache, kv):
    """Writes them into the pages of a layer's cache."""
    _, B, H, n, D = kv.shape
    pages = -(-n // PAGE)
    full = torch.zeros((2, B, H, pages * PAGE, D), dtype=kv.dtype, device=kv.device)
    full[:, :, :, :n] = kv
    full = full.view(2, B, H, pages, PAGE, D).permute(1, 3, 0, 2, 4, 5).reshape(B * pages, 2, H, PAGE, D)
    cache.pool[cache.page_table[:, :pages].reshape(-1).long()] = full


# ------------------------------------------------------------------------------------------ the framework's side
def _decoder(case, sd):
    m, L, n, B = MODELS[case["model"]], case["layers"], _max_len(case), case["rows"]
    if m["family"] == "gpt2":
        from poptransformer_b200 import gpt2
        return gpt2.GPT2Decoder(gpt2.GPT2Config(L, m["d"], m["heads"], m["vocab"], POSITIONS, n), sd, B)
    if m["family"] == "llama":
        from poptransformer_b200 import llama
        cfg = llama.LlamaConfig(L, m["d"], m["heads"], m["ffn"], m["vocab"], max_len=n, int4_group=case.get("group", 0))
        return llama.LlamaDecoder(cfg, sd, B, prefill=case["mode"] == "prompt")
    if m["family"] == "glm":
        from poptransformer_b200 import chatglm2
        cfg = chatglm2.ChatGLM2Config(L, m["d"], m["heads"], m["groups"], m["ffn"], m["vocab"], n, precision=case["weights"])
        return chatglm2.ChatGLM2Decoder(cfg, sd, B)
    if m["family"] == "rwkv":
        from poptransformer_b200 import rwkv
        return rwkv.RWKVDecoder(rwkv.RWKVConfig(L, m["d"], m["ffn"], m["vocab"], n), sd, B)
    from poptransformer_b200 import sabisun
    return sabisun.SabisunDecoder(sabisun.SabisunConfig(_sabisun_config(case), n), sd, B)


def prepare(case, seed):
    m, mode = MODELS[case["model"]], case["mode"]
    if mode == "products":
        from poptransformer_b200 import ops
        lins = [(ops.GemmWeight(ops.W_FP8, w, w_scale=ws), x, xs) for w, ws, x, xs in _products(case, seed)]
        return dict(case=case, ops=ops, lins=lins, workspace=ops.gemm_workspace(case["rows"], max(w.n_out for w, _, _ in lins)))
    dec = _decoder(case, _weights(case, seed))
    state = dict(case=case, dec=dec)
    if mode == "serve":
        state["prompts"], state["next"] = _requests(case, seed)
        return state
    n = {"decode": case["context"] + 1, "prompt": case["context"] + 1, "loop": case["context"]}[mode]
    ids = _ids(case, seed, n)
    state["ids"] = ids.pin_memory()
    dec.capture()
    if mode == "decode":
        if m["family"] == "sabisun":
            dec.reset(state["ids"])
            dec.prefill(case["context"])
        else:
            for i, cache in enumerate(dec.caches):
                _fill(cache, _history(case, seed, i, cache.n_kv, cache.head_dim))
    return state


def run(state):
    case, mode = state["case"], state["case"]["mode"]
    if mode == "products":
        ops = state["ops"]
        return [ops.gemm(ops.half_to_uint8(x, scale), w, x_scale=scale, workspace=state["workspace"]) for w, x, scale in state["lins"]]
    dec = state["dec"]
    if mode == "serve":
        seqs = [dec.open() for _ in state["prompts"]]
        out = [dec.extend([(s, p, [len(p) - 1]) for s, p in zip(seqs, state["prompts"])])]
        for tokens in state["next"]:
            out.append(dec.extend([(s, tokens[k:k + 1], [0]) for k, s in enumerate(seqs)]))
        for s in seqs:
            dec.close(s)
        return out
    if mode == "decode":
        dec.ids.copy_(state["ids"], non_blocking=True)
        dec.step_t.fill_(case["context"])
        dec.step()
        return {"logits": dec.logits, "ids": dec.ids}
    dec.reset(state["ids"])
    if mode == "prompt":
        dec.prefill()
        dec.step()
        return {"logits": dec.logits, "ids": dec.ids, "last cache": dec.caches[-1].pool}
    for _ in range(case["context"]):
        dec.step()
    return {"logits": dec.logits, "ids": dec.ids, "numerator": dec.st_num[-1], "denominator": dec.st_den[-1], "maximum": dec.st_max[-1]}


# ------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, w, eps=1e-5):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()


def _layer_norm(x, sd, key):
    return torch.nn.functional.layer_norm(x, x.shape[-1:], sd[key + ".weight"].double(), sd[key + ".bias"].double(), 1e-5)


def _attend(q, k, v, mask=None, scale=1.0, sink=None):
    """q [B, N, T, D], k / v [B, G, S, D]; mask [T, S] of what is hidden; sink [N]: one more logit in the denominator."""
    rep = q.shape[1] // k.shape[1]
    if rep > 1:
        k, v = k.repeat_interleave(rep, 1), v.repeat_interleave(rep, 1)
    s = (q @ k.transpose(-1, -2)) * scale
    if mask is not None:
        s = s.masked_fill(mask, -math.inf)
    if sink is not None:
        s = torch.cat([s, sink.double().view(1, -1, 1, 1).expand(s.shape[0], -1, s.shape[2], 1)], -1)
    p = torch.softmax(s, -1)
    return (p if sink is None else p[..., :-1]) @ v


def _half_tables(angle):
    a = angle.half().float()
    return torch.sin(a).half().double(), torch.cos(a).half().double()


def _heads(x, n):
    return x.view(*x.shape[:-1], n, -1).transpose(-3, -2)


def exact(case, seed):
    if case["mode"] == "products":
        return [((x.double() / xs).clamp(-448.0, 448.0).float().to(torch.float8_e4m3fn).double() @ w.view(torch.float8_e4m3fn).double().T) * (xs * ws)
                for w, ws, x, xs in _products(case, seed)]
    sd = _weights(case, seed)
    return {"gpt2": _gpt2_exact, "llama": _llama_exact, "glm": _glm_exact, "rwkv": _rwkv_exact, "sabisun": _sabisun_exact}[MODELS[case["model"]]["family"]](
        case, seed, MODELS[case["model"]], sd)


def _gpt2_exact(case, seed, m, sd):
    B, N, n = case["rows"], m["heads"], case["context"]
    x = sd["transformer.wte.weight"][_ids(case, seed, n + 1)[:, n].long().cuda()].double() + sd["transformer.wpe.weight"][n].double()

    def lin(key, x):
        return x @ sd[key + ".weight"].double().T + sd[key + ".bias"].double()

    for i in range(case["layers"]):
        p = f"transformer.h.{i}."
        q, k, v = (t.view(B, N, 1, -1) for t in lin(p + "attn.c_attn", _layer_norm(x, sd, p + "ln_1")).chunk(3, 1))
        old = _history(case, seed, i, N, m["d"] // N).double()
        a = _attend(q, torch.cat([old[0], k], 2), torch.cat([old[1], v], 2))
        x = x + lin(p + "attn.c_proj", a.reshape(B, -1))
        x = x + lin(p + "mlp.c_proj", torch.nn.functional.gelu(lin(p + "mlp.c_fc", _layer_norm(x, sd, p + "ln_2"))))
    return {"logits": _layer_norm(x, sd, "transformer.ln_f") @ sd["transformer.wte.weight"].double().T, "ids": None}


def _llama_exact(case, seed, m, sd):
    B, N, n, D = case["rows"], m["heads"], case["context"], m["d"] // m["heads"]
    ids, prompt = _ids(case, seed, n + 1), case["mode"] == "prompt"
    first = 0 if prompt else n
    x = sd["model.embed_tokens.weight"][ids[:, first:n + 1].long().cuda()].double()
    inv = torch.tensor([1.0 / 10000 ** (i / D) for i in range(0, D, 2)], device="cuda").half().float()
    sin, cos = _half_tables(torch.arange(first, n + 1, device="cuda").half().float()[:, None] * inv)
    sin, cos = torch.cat([sin, sin], -1), torch.cat([cos, cos], -1)
    hidden = torch.ones((n + 1, n + 1), dtype=torch.bool, device="cuda").triu(1) if prompt else None

    def weight(key):
        w = sd[key + ".weight"]
        if w.dtype != torch.int8:
            return w.double()
        q, s = torch.stack([w >> 4, (w << 4) >> 4], -1).view(w.shape[0], -1), sd[key + ".weight_scale"]
        return (q.view(*s.shape, -1).float() * s.float()[..., None]).half().double().view(q.shape)

    def lin(key, x):
        return x @ weight(key).T

    def turn(x):
        return x * cos + torch.cat([-x[..., D // 2:], x[..., :D // 2]], -1) * sin

    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, sd[p + "input_layernorm.weight"])
        q, k, v = (_heads(lin(p + f"self_attn.{c}_proj", h), N) for c in "qkv")
        q, k = turn(q), turn(k)
        if not prompt:
            old = _history(case, seed, i, N, D).double()
            k, v = torch.cat([old[0], k], 2), torch.cat([old[1], v], 2)
        a = _attend(q, k, v, hidden, D ** -0.5)
        x = x + lin(p + "self_attn.o_proj", a.transpose(1, 2).reshape(B, -1, m["d"]))
        h = _rms(x, sd[p + "post_attention_layernorm.weight"])
        x = x + lin(p + "mlp.down_proj", torch.nn.functional.silu(lin(p + "mlp.gate_proj", h)) * lin(p + "mlp.up_proj", h))
    out = {"logits": _rms(x[:, -1], sd["model.norm.weight"]) @ sd["lm_head.weight"].double().T, "ids": None}
    if prompt:
        pages = -(-_max_len(case) // PAGE)
        kv = torch.zeros((2, B, N, pages * PAGE, D), dtype=torch.float64, device="cuda")
        kv[0, :, :, :n + 1], kv[1, :, :, :n + 1] = k, v
        out["last cache"] = kv.view(2, B, N, pages, PAGE, D).permute(1, 3, 0, 2, 4, 5).reshape(B * pages, 2, N, PAGE, D)
    return out


def _glm_exact(case, seed, m, sd):
    B, N, G, n, D = case["rows"], m["heads"], m["groups"], case["context"], m["d"] // m["heads"]
    x = sd["transformer.embedding.word_embeddings.weight"][_ids(case, seed, n + 1)[:, n].long().cuda()].double()
    inv = torch.tensor([1.0 / 10000 ** (i / (D // 2)) for i in range(0, D // 2, 2)], dtype=torch.float32, device="cuda")
    sin, cos = _half_tables(n * inv)

    def lin(key, x, bias=False):
        y = x @ sd[key + ".weight"].double().T
        return y + sd[key + ".bias"].double() if bias else y

    def turn(x):
        e, o = x[..., 0:D // 2:2], x[..., 1:D // 2:2]
        return torch.cat([torch.stack([e * cos - o * sin, o * cos + e * sin], -1).flatten(-2), x[..., D // 2:]], -1)

    for i in range(case["layers"]):
        p = f"transformer.encoder.layers.{i}."
        h = _rms(x, sd[p + "input_layernorm.weight"])
        q = turn(lin(p + "self_attention.query", h, True).view(B, N, 1, D))
        k, v = lin(p + "self_attention.key_value", h, True).view(B, 2, G, 1, D).unbind(1)
        old = _history(case, seed, i, G, D).double()
        a = _attend(q, torch.cat([old[0], turn(k)], 2), torch.cat([old[1], v], 2), None, D ** -0.5)
        x = x + lin(p + "self_attention.dense", a.reshape(B, -1))
        h = _rms(x, sd[p + "post_attention_layernorm.weight"])
        x = x + lin(p + "mlp.dense_4h_to_h", torch.nn.functional.silu(lin(p + "mlp.dense_h_to_4h_1", h)) * lin(p + "mlp.dense_h_to_4h_2", h))
    return {"logits": lin("transformer.output_layer", _rms(x, sd["transformer.encoder.final_layernorm.weight"])), "ids": None}


def _rwkv_exact(case, seed, m, sd):
    B, d, L = case["rows"], m["d"], case["layers"]
    ids = _ids(case, seed, case["context"]).cuda()
    f64 = dict(dtype=torch.float64, device="cuda")
    st = [[torch.zeros((B, d), **f64) for _ in range(4)] + [torch.full((B, d), -1e30, **f64)] for _ in range(L)]

    def lin(key, x):
        return x @ sd[key + ".weight"].double().T

    def mix(t, key, old):
        w = sd[key].double().view(-1)
        return t * w + (1.0 - w) * old

    for t_ in range(case["context"]):
        x = sd["rwkv.embeddings.weight"][ids[:, t_].long()].double()
        for i in range(L):
            p, s = f"rwkv.blocks.{i}.", st[i]
            a, b = p + "attention.", p + "feed_forward."
            if i == 0:
                x = _layer_norm(x, sd, p + "pre_ln")
            t = _layer_norm(x, sd, p + "ln1")
            k, v, r = (lin(a + c, mix(t, a + "time_mix_" + c, s[1])) for c in ("key", "value", "receptance"))
            s[1] = t
            ww = k + sd[a + "time_first"].double()
            top = torch.maximum(s[4], ww)
            e1, e2 = torch.exp(s[4] - top), torch.exp(ww - top)
            wkv = (e1 * s[2] + e2 * v) / (e1 * s[3] + e2)
            ww = s[4] - torch.exp(sd[a + "time_decay"].double())
            top = torch.maximum(ww, k)
            e1, e2 = torch.exp(ww - top), torch.exp(k - top)
            s[2], s[3], s[4] = e1 * s[2] + e2 * v, e1 * s[3] + e2, top
            x = x + lin(a + "output", torch.sigmoid(r) * wkv)
            t = _layer_norm(x, sd, p + "ln2")
            k, r = (lin(b + c, mix(t, b + "time_mix_" + c, s[0])) for c in ("key", "receptance"))
            s[0] = t
            x = x + torch.sigmoid(r) * lin(b + "value", torch.relu(k) ** 2)
            if (i + 1) % 6 == 0:
                x = x / 2
        logits = lin("head", _layer_norm(x, sd, "rwkv.ln_out"))
    return {"logits": logits, "ids": None, "numerator": st[-1][2], "denominator": st[-1][3], "maximum": st[-1][4]}


def _sabisun_exact(case, seed, m, sd):
    cfg, L = _sabisun_config(case), case["layers"]
    if case["mode"] == "serve":
        prompts, more = _requests(case, seed)
        seqs = [np.concatenate([p, more[:, b]]) for b, p in enumerate(prompts)]
        wanted = [[len(p) - 1 + t for p in prompts] for t in range(1 + case["tokens"])]
    else:
        seqs = list(_ids(case, seed, case["context"] + 1).numpy()[:, :case["context"] + 1])
        wanted = [[case["context"]] * case["rows"]]
    T, B, W = max(map(len, seqs)), len(seqs), m["d"]
    ids = torch.zeros((B, T), dtype=torch.long)
    for b, s in enumerate(seqs):          # shorter ones are padded behind their end, where nothing looks
        ids[b, :len(s)] = torch.from_numpy(s.astype(np.int64))
    w = {k: v.double() for k, v in sd.items() if v.dim() == 1 or "hc" in k or "conv" in k}
    i, j = torch.arange(T, device="cuda")[:, None], torch.arange(T, device="cuda")
    hidden = (j > i) | ((i - j >= m["window"]) & (j >= m["keep_first"]))

    def lin(key, x):
        return x @ sd[key].double().T

    def attention(p, x, h):
        q, k, v = (_heads(lin(p + c, h), n) for c, n in (("q", x["heads"]), ("k", x["kv_heads"]), ("v", x["kv_heads"])))
        y = torch.cat([_attend(q[b:b + 1], k[b:b + 1], v[b:b + 1], hidden, x["scale"], w[p + "sink"]) for b in range(B)])
        return lin(p + "o", y.transpose(1, 2).reshape(B, T, -1))

    def mamba(p, x, h):
        H, P, S, G = x["heads"], x["vdim"], x["state"], x["groups"]
        inner = H * P
        z, u, dt = lin(p + "in", h).split([inner, inner + 2 * G * S, H], -1)
        u = torch.nn.functional.conv1d(torch.nn.functional.pad(u.transpose(1, 2), (x["conv"] - 1, 0)), w[p + "conv"][:, None], w[p + "conv.b"], groups=u.shape[-1])
        v, Bm, C = torch.nn.functional.silu(u.transpose(1, 2)).split([inner, G * S, G * S], -1)
        v, Bm, C = v.view(B, T, H, P), Bm.view(B, T, G, S).repeat_interleave(H // G, 2), C.view(B, T, G, S).repeat_interleave(H // G, 2)
        dt = torch.nn.functional.softplus(dt + w[p + "dt_bias"])
        keep = torch.exp(-torch.exp(w[p + "A_log"]) * dt)
        v_dt, state, y = v * dt[..., None], torch.zeros((B, H, S, P), dtype=torch.float64, device="cuda"), torch.empty_like(v)
        for t in range(T):
            state = torch.addcmul(state * keep[:, t, :, None, None], Bm[:, t, :, :, None], v_dt[:, t, :, None, :])
            y[:, t] = torch.matmul(C[:, t, :, None, :], state)[..., 0, :]
        g = (y + w[p + "D"][:, None] * v).reshape(B, T, inner) * torch.nn.functional.silu(z)
        g = g.view(B, T, x["norm_groups"], -1)
        return lin(p + "o", (g / torch.sqrt((g * g).mean(-1, keepdim=True) + 1e-5)).view(B, T, inner) * w[p + "norm"])

    xs = sd["embed"][ids.cuda()].double()[None].repeat(m["streams"], 1, 1, 1)
    for n in range(L):
        lay, p = cfg["layers"][n], f"l{n}."
        for q in "12":
            h = _rms(torch.tensordot(w[p + f"hc{q}.in"], xs, 1), w[p + "norm" + q])
            if q == "2":
                y = lin(p + "mlp.down", torch.relu(lin(p + "mlp.up", h)) ** 2)
            else:
                y = (attention if lay["type"] == "attention" else mamba)(p + "mix.", lay["mixer"], h)
            xs = torch.tensordot(w[p + f"hc{q}.mix"].T.contiguous(), xs, 1) + w[p + f"hc{q}.out"][:, None, None, None] * y
    x = _rms(xs.sum(0), w["final.norm"])
    out = [lin("embed", torch.stack([x[b, t] for b, t in enumerate(places)])) for places in wanted]
    return out if case["mode"] == "serve" else {"logits": out[0], "ids": None}


# ------------------------------------------------------------------------------------------ work and tolerance
def work(case):
    """Every weight once a step or pass (an embedding table's rows that are read apart), the history once, what is returned once."""
    m, L, B, n = MODELS[case["model"]], case["layers"], case["rows"], case["context"]
    d, V = m["d"], m["vocab"]
    per = {"int4": 0.5 + 2.0 / case.get("group", 128), "fp16": 2.0, "bf16": 2.0, "fp8": 1.0}[case["weights"]]
    head = V * d * (2.0 if case["weights"] == "int4" else per)
    if m["family"] == "rwkv":
        lin = L * (5 * d * d + 2 * d * m["ffn"])
        step = {"bytes": lin * per + head + B * (L * d * 2 * (3 * 4 + 2 * 2) + V * 2), "flops": 2.0 * B * (lin + V * d)}
        return {k: v * n for k, v in step.items()}
    if m["family"] == "sabisun":
        mamba, attn = L - L // 4, L // 4
        inner, kv = m["ssm_heads"] * 64, m["kv_heads"] * 128
        lin = mamba * d * (3 * inner + 2048 + m["ssm_heads"]) + attn * d * (2 * m["heads"] * 128 + 2 * kv) + 2 * L * d * m["ffn"]
        state, logits = mamba * m["ssm_heads"] * 64 * 128, V * 4
        if case["mode"] == "decode":
            keys = min(n + 1, m["window"] + m["keep_first"])
            return {"bytes": lin * 2 + V * d * 2 + B * (state * 8 + attn * keys * 2 * kv * 2 + logits),
                    "flops": 2.0 * B * (lin + V * d + 3 * state + attn * 2 * keys * m["heads"] * 128)}
        prompts, more = _requests(case, 0)
        T, steps = sum(map(len, prompts)), 1 + len(more)
        pairs = sum(sum(min(t + 1, m["window"] + m["keep_first"]) for t in range(len(p))) for p in prompts)
        toks = T + B * (steps - 1)
        return {"bytes": steps * (lin * 2 + V * d * 2 + B * (state * 4 + logits)) + (steps - 1) * B * state * 4 + attn * toks * 2 * kv * 2
                + (steps - 1) * attn * T * 2 * kv * 2,
                "flops": 2.0 * (toks * (lin + 3 * state) + steps * B * V * d + attn * 2 * (pairs + (steps - 1) * T) * m["heads"] * 128)}
    if case["mode"] == "products":
        kv, f = 2 * m["groups"] * (d // m["heads"]), m["ffn"]
        shapes = [(d + kv, d), (d, d), (2 * f, d), (d, f)] * L + [(V, d)]
        return {"bytes": float(sum(o * k + 2 * B * (o + k) for o, k in shapes)), "flops": 2.0 * B * sum(o * k for o, k in shapes)}
    kv = m.get("groups", m["heads"]) * (d // m["heads"])
    lin = L * {"gpt2": 12 * d * d, "llama": 4 * d * d + 3 * d * m.get("ffn", 0), "glm": 2 * d * d + 2 * kv * d + 3 * d * m.get("ffn", 0)}[m["family"]]
    if case["mode"] == "prompt":
        cache = L * B * (n + 1) * 2 * kv * 2
        return {"bytes": 2 * lin * per + head + 2 * cache + B * V * 2, "flops": 2.0 * (B * (n + 1) * lin + B * V * d + L * B * (n + 1) * (n + 2) * d)}
    return {"bytes": lin * per + head + L * B * (n + 1) * 2 * kv * 2 + B * V * 2, "flops": 2.0 * B * (lin + V * d + L * 2 * (n + 1) * d)}


def tolerance(case):
    """About four times what two orders of the sums of this path were measured to differ by: on INT4 logits 0.008 (largest 0.05) between
    the whole-step, per-matrix and tensor-memory forms, through the fp16 rounding after every operation of 32 blocks; on logits of bf16
    operands 0.01 from 64 bits; on single FP8 products only the fp16 rounding of the result.  A greedy id may turn where two logits are
    equal within that: one place of a row of the container."""
    return {"rel": {"int4": 0.03, "fp16": 0.02, "bf16": 0.03, "fp8": 0.001}[case["weights"]], "max": 0.2, "differ": 0.01}
