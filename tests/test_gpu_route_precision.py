"""Near-tie tokens of kleos_route_static on bf16 and of 16-bit training layers: probabilities and mCw come from 64-bit
logits.  Two experts, whose gate rows are alike but for one
small entry, and products of 2^8 that cancel: the fp32 sum loses about 2^-16 of the small difference, while the 64-bit
one keeps it.  mCw is the larger of two probabilities next to 1/2, so a 32-bit softmax of exact logits of
magnitude below 2^-7 is right to 2^-22: logits and their difference are exact to 2^-31, the exponentials near 1, their
sum, the quotient and the product are each rounded once or approximated to two units of 2^-24."""
import numpy as np
import pytest

from aristos_b200 import kleos, synth
from aristos_b200.config import KleosConfig
from tests import moe_harness as hz

pytestmark = pytest.mark.gpu


def _tokens(S, H):
    rng = np.random.default_rng(S)
    A, W = np.zeros((S, H), np.float32), np.zeros((2, H), np.float32)
    A[:, 0], A[:, 1] = 256.0, -256.0
    W[:, :2] = 1.0
    A[:, 2] = synth.round_to_dtype(rng.uniform(1.0, 2.0, S).astype(np.float32), 2)
    W[0, 2] = 2.0 ** -15          # the difference: 3e-5 to 6e-5
    A[:, 3] = synth.round_to_dtype(rng.uniform(-1.0, 1.0, S).astype(np.float32), 2)
    W[:, 3] = 2.0 ** -9           # common to both
    logits = A.astype(np.float64) @ W.astype(np.float64).T
    return A, W, 1.0 / (1.0 + np.exp(logits[:, 1] - logits[:, 0]))


def test_static():
    import torch
    S, H = 300, 256
    A, W, want = _tokens(S, H)
    Wp = np.zeros((64, H), np.float32)
    Wp[:2] = W
    a, w = (torch.from_numpy(x).cuda().bfloat16() for x in (A, Wp))
    probs = torch.empty(S, 64, dtype=torch.bfloat16, device="cuda")
    topk, mcw = torch.empty(S, 1, dtype=torch.int32, device="cuda"), torch.empty(S, device="cuda")
    kleos.route_static(a, w, None, S, H, 2, 1, 2, probs, topk, mcw)
    assert not topk.cpu().numpy().any()
    assert np.abs(mcw.cpu().numpy().astype(np.float64) - want).max() <= 2.0 ** -22


@pytest.mark.parametrize("dtype,train", [(2, 1), (3, 1)], ids=["bf16-training", "fp16-training"])
def test_layer(dtype, train):
    cfg = KleosConfig(sequence_len=256, hidden_size=256, intermediate_size=64, num_experts=2, expert_top_k=1,
                      torch_dtype=dtype, is_training=train, drop_tokens=0)
    packed, views = hz.make_inputs(cfg, 1)
    views[0]["A"][:], views[0]["Wg"][:2], want = _tokens(cfg.S, cfg.H)
    _, _, routing = hz.run_layer_single_gpu(cfg, packed[0])
    assert not routing["topk"].any()
    assert np.abs(routing["mcw"].astype(np.float64) - want).max() <= 2.0 ** -22


@pytest.mark.parametrize("H,E,K", [(640, 24, 8), (512, 16, 4), (2048, 64, 2)])
def test_mcw_is_no_less_exact_than_from_the_fp32_pipes(H, E, K):
    """mCw of the tensor-core router against 64 bits, and that of the FP32-pipe router on the same values."""
    import torch
    S = 4096
    rng = np.random.default_rng(H)
    A = synth.round_to_dtype(rng.standard_normal((S, H), dtype=np.float32), 2)
    W = np.zeros((64, H), np.float32)
    W[:E] = synth.round_to_dtype(rng.standard_normal((E, H), dtype=np.float32) / np.float32(np.sqrt(H)), 2)
    logits = A.astype(np.float64) @ W[:E].astype(np.float64).T
    p = np.exp(logits - logits.max(1, keepdims=True))
    want = -np.sort(-p, 1)[:, :K].sum(1) / p.sum(1)
    off = {}
    for dtype, tdt in ((0, torch.float32), (2, torch.bfloat16)):
        a, w = (torch.from_numpy(x).cuda().to(tdt) for x in (A, W))
        probs = torch.empty(S, 64, dtype=tdt, device="cuda")
        topk, mcw = torch.empty(S, K, dtype=torch.int32, device="cuda"), torch.empty(S, device="cuda")
        kleos.route_static(a, w, None, S, H, E, K, dtype, probs, topk, mcw)
        off[dtype] = np.sqrt((((mcw.cpu().numpy() - want) / want) ** 2).mean())
    assert off[2] <= off[0], off
