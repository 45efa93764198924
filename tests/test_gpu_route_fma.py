"""The FP32-pipe router at the edges of its blocks (32 tokens) and K split (sixteen values, eight warps),
and on logits that are not finite.  Expected: 64-bit logits and the selection rule of the oracle."""
import numpy as np
import pytest

from aristos_b200 import kleos, synth
from aristos_b200.config import KleosConfig
from oracle import moe_oracle
from tests import moe_harness as hz

pytestmark = pytest.mark.gpu


def _route(A, Wg, E, K, dtype):
    import torch
    S, H = A.shape
    w = np.zeros((64, H), np.float32)
    w[:E] = Wg
    tdt = torch.float32 if dtype == 0 else torch.uint16
    dev = [torch.from_numpy(synth.encode(x.ravel(), dtype)).view(tdt).cuda() for x in (A, w)]
    probs = torch.full((S * 64,), 7, dtype=tdt, device="cuda")
    topk = torch.full((S * K,), -5, dtype=torch.int32, device="cuda")
    mcw = torch.full((S,), -1.0, device="cuda")
    kleos.route_static(dev[0], dev[1], None, S, H, E, K, dtype, probs, topk, mcw)
    torch.cuda.synchronize()
    return topk.cpu().numpy().reshape(S, K), mcw.cpu().numpy(), synth.decode(probs.cpu().numpy(), dtype).reshape(S, 64)


@pytest.mark.parametrize("dtype", [0, 2])
@pytest.mark.parametrize("S,H,E,K", [(1, 64, 1, 1), (31, 64, 3, 2), (33, 192, 64, 8), (127, 1088, 33, 3), (2049, 448, 40, 2)])
def test_block_and_k_edges(S, H, E, K, dtype):
    rng = np.random.default_rng(S)
    A = synth.round_to_dtype(rng.standard_normal((S, H), dtype=np.float32), dtype)
    W = synth.round_to_dtype(rng.standard_normal((E, H), dtype=np.float32) / np.float32(np.sqrt(H)), dtype)
    topk, mcw, probs = _route(A, W, E, K, dtype)
    logits = A.astype(np.float64) @ W.astype(np.float64).T
    order = np.argsort(-logits, axis=1, kind="stable")[:, :K]
    assert np.array_equal(np.sort(topk, 1), np.sort(order, 1))
    p = np.exp(logits - logits.max(1, keepdims=True))
    p /= p.sum(1, keepdims=True)
    assert np.abs(probs[:, :E] - p).max() <= hz.PROB_TOL[dtype] and not probs[:, E:].any()
    assert np.abs(mcw - np.take_along_axis(p, order, 1).sum(1)).max() <= 1e-5


def test_logits_that_are_not_finite():
    """A NaN or -inf logit compares greater than nothing and is never chosen; places that stay empty hold id 0."""
    S, H, E, K = 40, 64, 4, 3
    A = np.zeros((S, H), np.float32)
    W = np.eye(E, H, dtype=np.float32)  # logit e = A[:, e]; W has zeros elsewhere
    A[:, :E] = [0.5, 2.0, -1.0, 1.0]
    A[1, 2] = np.inf     # inf * 0 = NaN in every other logit
    A[2, 0] = np.nan     # all logits NaN
    topk, mcw, probs = _route(A, W, E, K, 0)
    assert topk[0].tolist() == [1, 3, 0] and topk[39].tolist() == [1, 3, 0]
    assert topk[1].tolist() == [2, 0, 0] and topk[2].tolist() == [0, 0, 0]
    assert np.isnan(mcw[[1, 2]]).all() and np.isnan(probs[2, :E]).all()


@pytest.mark.parametrize("kw", [dict(num_experts=256, torch_dtype=2), dict(num_experts=256, torch_dtype=1),
                                dict(num_experts=96, torch_dtype=0, is_training=1)], ids=["bf16-256", "tf32-256", "float-96-training"])
def test_wide_layers(kw):
    cfg = KleosConfig(sequence_len=512, hidden_size=256, intermediate_size=128, **kw)
    packed, views = hz.make_inputs(cfg, 1)
    ref = moe_oracle.moe_forward(cfg, 1, views)[0]
    probs, out, routing = hz.run_layer_single_gpu(cfg, packed[0], forwards=2)
    hz.check_against_oracle(cfg, ref, probs, out, routing)


@pytest.mark.parametrize("E,kw", [(129, dict(torch_dtype=0, is_training=1)), (160, dict(torch_dtype=2)), (176, dict(torch_dtype=1, is_training=1)),
                                  (192, dict(torch_dtype=3, expert_top_k=8))], ids=["129-float-training", "160-bf16", "176-tf32-training", "192-fp16"])
def test_three_column_tiles(E, kw):
    """129 to 192 experts."""
    cfg = KleosConfig(sequence_len=384, hidden_size=256, intermediate_size=128, num_experts=E, **kw)
    packed, views = hz.make_inputs(cfg, 1)
    ref = moe_oracle.moe_forward(cfg, 1, views)[0]
    probs, out, routing = hz.run_layer_single_gpu(cfg, packed[0], forwards=2)
    hz.check_against_oracle(cfg, ref, probs, out, routing)
    if not cfg.is_training:
        return
    import torch
    info = kleos.initialize(cfg, 0, 1)
    try:
        iP, oP = torch.from_numpy(packed[0]).cuda(), torch.zeros(info.output_elems, device="cuda")
        kleos.forward_host(iP, oP)
        st = kleos.gate_stats(info)
    finally:
        kleos.finalize()
    assert np.array_equal(st["mean_count"], ref["counts"].astype(np.float32) / np.float32(cfg.S))
    assert np.abs(st["mean_prob"] - ref["mean_prob"]).max() <= 2e-6
