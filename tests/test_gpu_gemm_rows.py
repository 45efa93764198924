"""Expert GEMM of 16-bit and TF32 layers at the row counts where its tiles change: remainders of 16 and 32
rows, one tile of up to 288 rows, several of up to 256, experts without rows; more tiles than block pairs,
so that the ring of accumulators wraps around; columns that end inside a tile."""
import numpy as np
import pytest

from aristos_b200 import synth
from aristos_b200.config import KleosConfig
from oracle import moe_oracle
from tests import moe_harness as hz

pytestmark = pytest.mark.gpu

ROWS = {
    "few": [1, 15, 16, 0, 17, 33, 255, 256, 257, 288, 289],
    "many": [512, 513, 545, 577, 0, 31],
}


@pytest.mark.parametrize("dtype", [1, 2, 3])
@pytest.mark.parametrize("name,I,act", [("few", 4160, 0), ("few", 448, 1), ("many", 4160, 1), ("many", 320, 0)])
def test_rows_of_an_expert(name, I, act, dtype):
    rows = list(ROWS[name])
    S = -(-(sum(rows) + 1) // 128) * 128
    rows.append(S - sum(rows))
    E = len(rows)
    cfg = KleosConfig(sequence_len=S, hidden_size=192, intermediate_size=I, num_experts=E, expert_top_k=1, torch_dtype=dtype,
                      hidden_act=act, **(dict(capacity_factor=2.4) if name == "few" else dict(drop_tokens=0)))
    assert max(rows) <= cfg.EC
    packed, views = hz.make_inputs(cfg, 1, bias_scale=0.5)
    # tokens that lean on one expert's gate row, in mixed order: expert e gets rows[e] of them
    rng = np.random.default_rng(S)
    expert = rng.permutation(np.repeat(np.arange(E), rows))
    Wg = views[0]["Wg"][:E]
    tokens = 0.3 * rng.standard_normal((S, cfg.H)) + 6.0 * Wg[expert] / (Wg[expert] ** 2).sum(1, keepdims=True)
    views[0]["A"][:] = synth.round_to_dtype(tokens.astype(np.float32).ravel(), dtype).reshape(S, cfg.H)
    ref = moe_oracle.moe_forward(cfg, 1, views)[0]
    assert np.array_equal(ref["counts"], rows)
    probs, out, routing = hz.run_layer_single_gpu(cfg, packed[0], forwards=2)
    hz.check_against_oracle(cfg, ref, probs, out, routing)


@pytest.mark.parametrize("S", [128, 384, 4096])
def test_rows_of_the_dense_layer(S):
    import torch
    cfg = KleosConfig(sequence_len=S, hidden_size=192, intermediate_size=320, num_experts=1, expert_top_k=1, torch_dtype=2)
    packed, views = hz.make_inputs(cfg, 1, bias_scale=0.5)
    _, out, _ = hz.run_layer_single_gpu(cfg, packed[0], forwards=2)
    v = {k: torch.from_numpy(np.ascontiguousarray(x)).double() for k, x in views[0].items() if x.size}
    y = torch.relu(v["A"] @ v["W1"][0].T + v["b1"][0])
    want = (y @ v["W2"][0].T + v["b2"][0]).numpy()
    assert np.abs(out - want).max() <= hz.TOL[2] * np.abs(want).max()
