"""Norms where the number of units a thread has, the order in which gains are read or the blocks an SM takes change with rows and width, against the oracle."""
import numpy as np
import pytest
import torch

from oracle import ops_np as O
from poptransformer_b200 import ops

pytestmark = pytest.mark.gpu


def _some(rows):
    return sorted({0, min(1, rows - 1), rows // 2, rows - 1})


def _bound(exp, beta):
    """Another order of the fp32 sums may move the rounded mean (of at most a few tenths, for eight elements one) and inverse deviation by an ulp, and the roundings
    of product, gain and offset behind them by one each."""
    return 4 * 2.0 ** -10 * (np.abs(exp) + np.abs(beta.astype(np.float32)) + 4)


# one, two and four units a thread, ragged last units, one row; more blocks than SMs hold at once
@pytest.mark.parametrize("rows,dim", [(2, 8), (3, 2048), (3, 2056), (150, 2056), (297, 1600), (592, 4096), (593, 4096), (612, 8184), (5000, 1000), (5001, 1000), (2, 8184)])
def test_norm_ce(cuda, rows, dim):
    r = np.random.default_rng(rows + dim)
    x, g, b = r.standard_normal((rows, dim)).astype(np.float16), (1 + 0.1 * r.standard_normal(dim)).astype(np.float16), (0.1 * r.standard_normal(dim)).astype(np.float16)
    got = ops.layer_norm_ce(*(torch.from_numpy(t).to(cuda) for t in (x, g, b)), 1e-5).cpu().numpy()
    some = _some(rows)
    exp = O.norm_ce(x[some], g, b, 1e-5).astype(np.float32)
    assert (np.abs(got[some].astype(np.float32) - exp) <= _bound(exp, b)).all() and np.isfinite(got.astype(np.float32)).all()


@pytest.mark.parametrize("rows,dim", [(3, 4096), (3, 4104), (600, 512), (1000, 4096), (488, 8184), (490, 8184)])
def test_norm_mix(cuda, rows, dim):
    """The mixes of the normalised row, bit by bit those of the two launches they stand for."""
    L, P, S = ops._lib.lib(), ops._ptr, ops._stream
    gen = torch.Generator(device=cuda).manual_seed(rows + dim)
    rand = lambda *s: torch.randn(s, generator=gen, device=cuda).half()
    x, state, g, b, w = rand(rows, dim), rand(rows, dim), rand(dim), rand(dim), [torch.rand(dim, generator=gen, device=cuda).half() for _ in range(3)]
    outs, kept = [torch.empty_like(x) for _ in range(3)], state.clone()
    ops.check(L.pt_norm_ce_mix(P(x), P(g), P(b), rows, dim, 1e-5, P(kept), *map(P, w), *map(P, outs), S()), "mix")
    h = kept                                                    # (the state takes the normalised row)
    one = torch.ones((), dtype=torch.float16, device=cuda)
    for o, m in zip(outs, w):
        assert torch.equal(o, h * m + (one - m) * state)
    some = _some(rows)
    exp = O.norm_ce(x[some].cpu().numpy(), g.cpu().numpy(), b.cpu().numpy(), 1e-5).astype(np.float32)
    assert (np.abs(h[some].cpu().numpy().astype(np.float32) - exp) <= _bound(exp, b.cpu().numpy())).all()


@pytest.mark.parametrize("rows,dim", [(1, 8), (2, 2056), (149, 4096), (297, 1600), (592, 2048), (593, 8184), (3, 16384)])
@pytest.mark.parametrize("residual", [False, True])
def test_rms_norm(cuda, rows, dim, residual):
    r = np.random.default_rng(rows + dim)
    x, res, g = (r.standard_normal(s).astype(np.float16) for s in ((rows, dim), (rows, dim), (dim,)))
    some = _some(rows)
    t = [torch.from_numpy(v).to(cuda) for v in (x, g)]
    got = ops.rms_norm(*t, 1e-5, residual=torch.from_numpy(res).to(cuda)) if residual else ops.rms_norm(*t, 1e-5)
    h = x[some]
    if residual:
        got, s = got
        h = O.add_f16(x[some], res[some])
        assert np.array_equal(s.cpu().numpy()[some].view(np.uint16), h.view(np.uint16))
    exp = O.rms_norm(h, g, 1e-5).astype(np.float32)
    # another order of the fp32 sums: an ulp of the rounded inverse, and one of the two roundings behind it
    assert (np.abs(got.cpu().numpy()[some].astype(np.float32) - exp) <= 3 * 2.0 ** -10 * np.abs(exp) + 2.0 ** -24).all()
