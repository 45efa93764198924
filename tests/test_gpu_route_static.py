"""kleos_route_static on bf16 where its accumulators are filled more than once (an accumulator per 64 values of K,
eight at a time, four blocks per 128 tokens: from H = 2112 on), and on logits that are not finite."""
import numpy as np
import pytest

from aristos_b200 import kleos, synth
from tests import moe_harness as hz

pytestmark = pytest.mark.gpu


def _route(A, Wg, K, bias=None):
    import torch
    (S, H), E = A.shape, len(Wg)
    w = np.zeros((64, H), np.float32)
    w[:E] = Wg
    a, w = (torch.from_numpy(x).cuda().bfloat16() for x in (A, w))
    b = None if bias is None else torch.from_numpy(np.asarray(bias, np.float32)).cuda()
    probs = torch.full((S, 64), 7, dtype=torch.bfloat16, device="cuda")
    topk = torch.full((S, K), -5, dtype=torch.int32, device="cuda")
    mcw = torch.full((S,), -1.0, device="cuda")
    for _ in range(2):
        kleos.route_static(a, w, b, S, H, E, K, 2, probs, topk, mcw)
    return topk.cpu().numpy(), mcw.cpu().numpy(), probs.float().cpu().numpy()


@pytest.mark.parametrize("S,H,E,K", [
    (300, 2112, 64, 2),    # 33 slices: one block of the four fills its accumulators twice
    (200, 2112, 24, 3),
    (129, 4096, 64, 3),    # 16 slices a block: twice everywhere
    (300, 4096, 8, 2),
    (77, 6208, 33, 8),     # 24 and 25: three and four times
    (385, 6208, 64, 2),
])
def test_accumulators_filled_again(S, H, E, K):
    rng = np.random.default_rng(H + K)
    A = synth.round_to_dtype(rng.standard_normal((S, H), dtype=np.float32), 2)
    W = synth.round_to_dtype(rng.standard_normal((E, H), dtype=np.float32) / np.float32(np.sqrt(H)), 2)
    topk, mcw, probs = _route(A, W, K)
    logits = A.astype(np.float64) @ W.astype(np.float64).T
    order = np.argsort(-logits, axis=1, kind="stable")[:, :K]
    assert np.array_equal(np.sort(topk, 1), np.sort(order, 1))
    p = np.exp(logits - logits.max(1, keepdims=True))
    p /= p.sum(1, keepdims=True)
    assert np.abs(probs[:, :E] - p).max() <= hz.PROB_TOL[2] and not probs[:, E:].any()
    assert np.abs(mcw - np.take_along_axis(p, order, 1).sum(1)).max() <= 1e-5


def test_logits_that_are_not_finite():
    """A NaN or -inf logit compares greater than nothing and is never chosen; places that stay empty hold id 0."""
    S, H, E, K = 140, 256, 4, 3
    A, W = np.zeros((S, H), np.float32), np.eye(E, H, dtype=np.float32)  # logit e = A[:, e]
    A[:, :E] = [0.5, 2.0, -1.0, 1.0]
    A[1, 2] = np.inf     # inf * 0 = NaN in every other logit
    A[130, 0] = np.nan   # all logits NaN
    topk, mcw, probs = _route(A, W, K)
    assert topk[1].tolist() == [2, 0, 0] and topk[130].tolist() == [0, 0, 0]
    assert np.isnan(mcw[[1, 130]]).all() and np.isnan(probs[130, :E]).all()
    finite = ~np.isin(np.arange(S), [1, 130])
    assert (topk[finite] == [1, 3, 0]).all() and np.isfinite(mcw[finite]).all()


def test_an_expert_masked_by_an_infinite_bias():
    S, H, E, K = 130, 128, 3, 2
    A, W = np.zeros((S, H), np.float32), np.eye(E, H, dtype=np.float32)
    A[:, :E] = [1.0, 4.0, 2.0]
    topk, mcw, probs = _route(A, W, K, bias=[0.0, -np.inf, 0.0])
    assert (topk == [2, 0]).all() and not probs[:, 1].any()
    assert np.abs(mcw - 1.0).max() <= 2.0 ** -22   # both others: exponentials over their own sum
