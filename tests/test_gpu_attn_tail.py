"""Decode attention where one early key has by far the highest score: the many others still count, each as exactly as fp16 weights allow."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# few (row, kv head) pairs, whose keys are spread over many warps, and many, where four warps take all of a pair's
@pytest.mark.parametrize("B", [1, 40, 150])
@pytest.mark.parametrize("H", [64, 128])
@pytest.mark.parametrize("below", [8.0, 12.0, 14.5, 17.5, 19.5])
def test_flat_tail_behind_a_spike(cuda, B, H, below):
    from poptransformer_b200 import ops
    N, G, n = 2, 2, 2000
    g = torch.Generator(device=cuda).manual_seed(B + H)
    cache = ops.PagedKVCache(B, G, H, 2048, 64, cuda)
    pool = cache.pool.view(B, -1, 2, G, 64, H)
    # scores are exact: q is a unit vector, and the keys' first channel is the score
    pool[:, :, 0] = 0
    pool[:, :, 0, ..., 0] = -below
    pool[:, 0, 0, :, 3, 0] = 0
    pool[:, :, 1] = torch.rand(pool[:, :, 1].shape, generator=g, device=cuda).half() * 0.5 + 0.5
    pool[:, 0, 1, :, 3] = 0                                   # all of the output is the tail's
    qkv = torch.zeros((B, (N + 2 * G), H), dtype=torch.float16, device=cuda)
    qkv[:, :N, 0] = 1
    qkv[:, N:N + G, 0] = -below
    qkv[:, N + G:] = 0.75
    V = pool[:, :, 1].permute(0, 2, 1, 3, 4).reshape(B, G, -1, H)[:, :, :n].double()
    tail = V.sum(2) + 0.75                                     # (the spike's value is zero)
    w = torch.exp(torch.tensor(-below, dtype=torch.float64, device=cuda))
    exp = (w * tail / (1 + n * w)).reshape(B, G * H)
    got = ops.kv_append_attn(qkv.view(B, -1), torch.full((1,), n, dtype=torch.int32, device=cuda), cache, N, score_scale=1.0).double()
    # weights and output are rounded to fp16 once (the output may be below its normal numbers), the fp32 sums lose 2^-23 a key
    bound = exp * (2 * 2.0 ** -11 + n * 2.0 ** -23) + 2.0 ** -25
    assert bool(((got - exp).abs() <= bound).all()), float(((got - exp).abs() / bound).max())
