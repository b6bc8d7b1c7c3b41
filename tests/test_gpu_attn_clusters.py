"""Decode attention where the blocks of a cluster share a (row, kv head) pair's keys, and at the edges of the chunks that a warp takes."""
import pytest
import test_gpu_attn_pages

pytestmark = pytest.mark.gpu


# (rows, q heads, kv heads, head width, page size, pages): clusters of 2, 4 (a part of the q heads per unit), 8 and 16 blocks, the last with
# pages of 8, where a chunk has rows of several pages; blocks of 8 warps with less keys than warps
@pytest.mark.parametrize("B,N,G,H,page,pages", [(5, 12, 12, 64, 64, 17), (2, 24, 2, 128, 24, 50), (2, 8, 8, 128, 64, 40), (1, 8, 2, 128, 8, 300), (1, 4, 4, 64, 16, 20)])
@pytest.mark.parametrize("softmax", ["f32", "f16"])
def test_clusters(cuda, B, N, G, H, page, pages, softmax):
    test_gpu_attn_pages.test_runs_of_pages(cuda, B, N, G, H, page, pages, softmax)


@pytest.mark.parametrize("mode", ["llama", "chatglm2"])
@pytest.mark.parametrize("aligned", [True, False])
def test_rotation_tables_anywhere(cuda, mode, aligned):
    """The tables may begin off 16-byte boundaries; the cached key and the output are those of tables that do not."""
    import torch
    from poptransformer_b200 import ops
    g = torch.Generator(device=cuda).manual_seed(3)
    B, N, G, H, L = 2, 8, 2, 128, 100
    half = H // 2 if mode == "llama" else H // 4
    tables = [torch.rand((L, half), device=cuda, generator=g).half() for _ in range(2)]
    qkv = torch.randn((B, (N + 2 * G) * H), device=cuda, generator=g).half() * 0.5
    got = []
    for off in (0, 0 if aligned else 1):
        bufs = [torch.empty(t.numel() + 8, dtype=torch.float16, device=cuda)[off:off + t.numel()].view_as(t).copy_(t) for t in tables]
        cache = ops.PagedKVCache(B, G, H, L, 64, cuda)
        cache.pool.fill_(0.25)
        out = ops.kv_append_attn(qkv, torch.full((1,), 70, dtype=torch.int32, device=cuda), cache, N, rope_mode=ops.ROPE_LLAMA if mode == "llama" else ops.ROPE_CHATGLM2,
                                 score_scale=0.088, rope_sin=bufs[0], rope_cos=bufs[1])
        got.append((out, cache.pool.clone()))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
