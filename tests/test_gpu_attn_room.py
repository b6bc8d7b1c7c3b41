"""Decode attention of a short history in a table with much room behind it: as many blocks share the work as the history has pages."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _runs(ws, rows, heads, pages):
    """How many runs of pages left results in the workspace ([counters][(max, sum) per head and run] ...), for every (row, head)."""
    off = -(-rows * heads * 4 // 256) * 256
    ml = ws[off:off + rows * heads * pages * 8].view(torch.float32).view(rows * heads, pages, 2)
    return (~torch.isnan(ml[:, :, 1])).sum(1)


# (rows, q heads, kv heads, pages of the table): 32 and 128 (row, kv head) pairs, and two of more than the SMs hold at a time
@pytest.mark.parametrize("B,N,G,pages", [(8, 32, 2, 64), (4, 32, 32, 64), (4, 32, 32, 512), (20, 32, 32, 100), (1, 8, 8, 33)])
@pytest.mark.parametrize("used", [1, 2, 8, 31, 33])
def test_history_shared_by_blocks(cuda, B, N, G, pages, used):
    from poptransformer_b200 import ops
    page, H = 64, 128
    g = torch.Generator(device=cuda).manual_seed(B * pages + used)
    # rows share one pool of `used` pages each; the other entries of the table are never read
    table = torch.full((B, pages), 1 << 30, dtype=torch.int32, device=cuda)
    table[:, :used] = torch.randperm(B * used, generator=g, device=cuda).to(torch.int32).view(B, used)
    cache = ops.PagedKVCache(B, G, H, page * pages, page, cuda, page_table=table, n_pages=B * used)
    step = page * (used - 1) + 5
    hist = torch.randn((2, B, G, used * page, H), device=cuda, generator=g).half() * 0.5
    old = hist.clone()
    old[:, :, :, step:] = float("nan")
    cache.pool[table[:, :used].long().reshape(-1)] = old.view(2, B, G, used, page, H).permute(1, 3, 0, 2, 4, 5).reshape(B * used, 2, G, page, H)
    qkv = torch.randn((B, (N + 2 * G) * H), device=cuda, generator=g).half() * 0.5
    q, k, v = qkv.double().split([N * H, G * H, G * H], 1)
    K = torch.cat([hist[0, :, :, :step].double(), k.view(B, G, 1, H)], 2).repeat_interleave(N // G, 1)
    V = torch.cat([hist[1, :, :, :step].double(), v.view(B, G, 1, H)], 2).repeat_interleave(N // G, 1)
    s = (q.view(B, N, 1, H) @ K.transpose(-1, -2)) / math.sqrt(H)
    exp = (torch.softmax(s, -1) @ V).view(B, N * H)
    ws, err = ops.attn_workspace(B, N, H, pages, cuda), torch.zeros(1, dtype=torch.int32, device=cuda)
    ws[-(-B * N * 4 // 256) * 256:].view(torch.float32).fill_(float("nan"))
    got = ops.kv_append_attn(qkv, torch.full((1,), step, dtype=torch.int32, device=cuda), cache, N, score_scale=float(np.float16(1 / math.sqrt(H))), workspace=ws, error_flag=err)
    bound = (4 * 2.0 ** -11 * (1 + s.abs().amax(-1).view(B, N, 1)) * V.abs().amax(2)).view(B, N * H)      # scores twice, weights and output once rounded to fp16
    assert bool(((got.double() - exp).abs() <= bound).all()) and int(err.item()) == 0 and int(ws[:B * N * 4].count_nonzero()) == 0
    units = B * G * -(-(N // G) // 8)
    runs = _runs(ws, B, N, pages)
    least = min(used, max(1, 4 * torch.cuda.get_device_properties(cuda).multi_processor_count // units))
    # dealing `used` pages out to r blocks evenly leaves at least half of min(used, r) blocks with pages; a single run writes the output itself
    assert int(runs.min()) == int(runs.max()) and max(1, int(runs.min())) >= (least + 1) // 2
