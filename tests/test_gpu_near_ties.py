"""Near-tie selection with logits on the edge of the band around the k-th one.  Tokens of zeros have the gate
bias as their logits, in every arithmetic, so the edge can be hit to the bit: the experts that come first here
are further above the k-th logit than the band is wide, while the rounded sum of the two is not below them."""
import numpy as np
import pytest

from aristos_b200 import kleos, synth
from aristos_b200.config import KleosConfig
from tests import moe_harness as hz

pytestmark = pytest.mark.gpu

F = np.float32
EDGE = {
    "second of two": ([F(1.0001), F(1.0), F(0.99995)], 2),
    "at one half": ([F(0.5) + F(1678 * 2.0 ** -24), F(0.5), F(0.49995)], 2),
    "two on the edge": ([F(1.0001), F(1.0001), F(1.0), F(0.99995)], 3),
}


def _bias(name, E):
    lead, K = EDGE[name]
    eps = F(1e-4) * max(F(1), abs(lead[K - 1]))
    assert lead[0] - lead[K - 1] > eps and not lead[0] > lead[K - 1] + eps and lead[K - 1] - lead[K] < eps
    return np.array(list(lead) + [F(0)] * (E - len(lead)), F), K


@pytest.mark.parametrize("name", EDGE)
def test_edge_of_the_band_static(name):
    import torch
    S, H, E = 200, 256, 8
    bias, K = _bias(name, E)
    A = torch.zeros(S, H, dtype=torch.bfloat16, device="cuda")
    Wg = torch.ones(64, H, dtype=torch.bfloat16, device="cuda")
    probs = torch.empty(S, 64, dtype=torch.bfloat16, device="cuda")
    topk = torch.empty(S, K, dtype=torch.int32, device="cuda")
    mcw = torch.empty(S, device="cuda")
    kleos.route_static(A, Wg, torch.from_numpy(bias).cuda(), S, H, E, K, 2, probs, topk, mcw)
    assert (np.sort(topk.cpu().numpy(), 1) == np.arange(K)).all()


@pytest.mark.parametrize("name", EDGE)
@pytest.mark.parametrize("dtype,train,flow", [(2, 0, "0"), (3, 1, "0"), (1, 0, "0"), (0, 0, "0"), (2, 0, "1")],
                         ids=["bf16", "fp16-training", "tf32", "float", "bf16-persistent"])
def test_edge_of_the_band_layer(name, dtype, train, flow, monkeypatch):
    monkeypatch.setenv("KLEOS_FLOW", flow)
    bias, K = _bias(name, 8)
    cfg = KleosConfig(sequence_len=256, hidden_size=128, intermediate_size=64, num_experts=8, expert_top_k=K,
                      torch_dtype=dtype, is_training=train, drop_tokens=0)
    packed, views = hz.make_inputs(cfg, 1)
    views[0]["A"][:] = 0.0
    _, _, routing = hz.run_layer_single_gpu(cfg, packed[0], gate_bias=bias)
    assert (np.sort(routing["topk"], 1) == np.arange(K)).all()
    assert np.array_equal(routing["counts"], [cfg.S] * K + [0] * (8 - K))
