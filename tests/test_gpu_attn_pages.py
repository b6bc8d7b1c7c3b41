"""Attention kernels at the sizes where their split of the pages changes, against float64."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# (rows, q heads, kv heads, head width, page size, pages): as many (row, kv head) pairs that a block walks several pages, up to all of them (a
# table of 11 or 5 pages) or to a part whose results are combined (30, 20); 16 q heads per kv head; pages of 16, 64 and 128.
@pytest.mark.parametrize("B,N,G,H,page,pages", [(16, 32, 32, 128, 64, 11), (40, 8, 8, 64, 16, 30), (24, 32, 2, 128, 64, 20), (16, 16, 16, 128, 128, 5), (7, 12, 12, 64, 64, 90)])
@pytest.mark.parametrize("softmax", ["f32", "f16"])
def test_runs_of_pages(cuda, B, N, G, H, page, pages, softmax):
    """One step on top of a random history at positions around the edges of pages and of runs; the pool is NaN wherever no token is."""
    from poptransformer_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(B * pages)
    cache = ops.PagedKVCache(B, G, H, page * pages, page, cuda)
    cache.page_table.copy_(torch.randperm(B * pages, generator=g, device=cuda).to(torch.int32).view(B, pages))
    ws, err = ops.attn_workspace(B, N, H, pages, cuda), torch.zeros(1, dtype=torch.int32, device=cuda)
    L = page * pages
    hist = torch.randn((2, B, G, L, H), device=cuda, generator=g).half() * 0.5
    table = cache.page_table.long()
    for step in sorted({0, page - 1, page, 2 * page, 3 * page + 5, (pages // 2) * page - 1, (pages // 2) * page, L - page, L - 1}):
        cache.pool.fill_(float("nan"))
        old = hist.clone()
        old[:, :, :, step:] = float("nan")
        cache.pool[table.reshape(-1)] = old.view(2, B, G, pages, page, H).permute(1, 3, 0, 2, 4, 5).reshape(B * pages, 2, G, page, H)
        qkv = torch.randn((B, (N + 2 * G) * H), device=cuda, generator=g).half() * 0.5
        q, k, v = qkv.double().split([N * H, G * H, G * H], 1)
        K = torch.cat([hist[0, :, :, :step].double(), k.view(B, G, 1, H)], 2).repeat_interleave(N // G, 1)
        V = torch.cat([hist[1, :, :, :step].double(), v.view(B, G, 1, H)], 2).repeat_interleave(N // G, 1)
        s = (q.view(B, N, 1, H) @ K.transpose(-1, -2)) / math.sqrt(H)
        exp = (torch.softmax(s, -1) @ V).view(B, N * H)
        got = ops.kv_append_attn(qkv, torch.full((1,), step, dtype=torch.int32, device=cuda), cache, N, softmax_mode=ops.SOFTMAX_F32 if softmax == "f32" else ops.SOFTMAX_F16,
                                 score_scale=float(np.float16(1 / math.sqrt(H))), workspace=ws, error_flag=err)
        # scores are rounded to fp16 twice (2^-11 of up to |s|), weights and the output once, in f16 mode the weights twice
        bound = (4 * 2.0 ** -11 * (1 + s.abs().amax(-1).view(B, N, 1)) * V.abs().amax(2)).view(B, N * H)
        assert bool(((got.double() - exp).abs() <= bound).all()), step
        page_of, slot = table[:, step // page], step % page
        assert torch.equal(cache.pool[page_of, 0, :, slot], k.view(B, G, H).half()) and torch.equal(cache.pool[page_of, 1, :, slot], v.view(B, G, H).half())
    assert int(err.item()) == 0 and int(ws[:B * N * 4].count_nonzero()) == 0


def test_prompt_rows_off_16_byte_boundaries(cuda):
    """The rotation reads and writes element by element where rows are not on 16-byte boundaries: the same bits as where they are."""
    from poptransformer_b200 import ops
    from poptransformer_b200.llama import rope_tables
    B, P, N, H = 2, 70, 3, 128
    sin, cos = rope_tables(128, H, cuda)
    base = torch.randn((B * P, 3 * N * H), device=cuda).half()
    outs = []
    for off in (0, 2):
        buf = torch.empty(base.numel() + 8, dtype=torch.float16, device=cuda)
        qkv = buf[off:off + base.numel()].view_as(base)
        qkv.copy_(base)
        cache = ops.PagedKVCache(B, N, H, 128, 64, cuda)
        out = ops.prefill_attn(qkv, cache, B, P, 0, N, 0.09, sin, cos)
        outs.append((out, qkv.clone(), cache.pool))
    assert all(torch.equal(a, b) for a, b in zip(*outs))
