"""The documented switches of the router and of the row gathering: KLEOS_ROUTE_KERNELS=1 (the separate router kernels
for 16-bit and TF32 layers of up to 128 experts) and KLEOS_GATHER=0 (rows copied into the cells at any size)."""
import numpy as np
import pytest

from aristos_b200.config import KleosConfig
from oracle import moe_oracle
from tests import moe_harness as hz

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,H,E,K,dtype,train", [
    (384, 192, 33, 2, 2, 0),
    (256, 320, 64, 8, 3, 1),
    (128, 64, 3, 2, 1, 0),
    (384, 448, 100, 4, 2, 1),
    (256, 192, 128, 2, 1, 1),
], ids=lambda v: str(v))
def test_separate_router_kernels(S, H, E, K, dtype, train, monkeypatch):
    monkeypatch.setenv("KLEOS_ROUTE_KERNELS", "1")
    cfg = KleosConfig(sequence_len=S, hidden_size=H, intermediate_size=64, num_experts=E, expert_top_k=K, torch_dtype=dtype, is_training=train)
    packed, views = hz.make_inputs(cfg, 1, bias_scale=0.5)
    ref = moe_oracle.moe_forward(cfg, 1, views)[0]
    probs, out, routing = hz.run_layer_single_gpu(cfg, packed[0], forwards=2)
    hz.check_against_oracle(cfg, ref, probs, out, routing)


@pytest.mark.parametrize("S,H,I,E,K,dtype", [
    (256, 512, 320, 8, 2, 2),       # 64 rows an expert
    (512, 192, 448, 16, 8, 3),      # 256: the most that are gathered
    (384, 128, 192, 100, 1, 1),     # experts without rows
], ids=lambda v: str(v))
def test_gathered_and_copied_rows_give_the_same_bits(S, H, I, E, K, dtype, monkeypatch):
    cfg = KleosConfig(sequence_len=S, hidden_size=H, intermediate_size=I, num_experts=E, expert_top_k=K, torch_dtype=dtype)
    packed, _ = hz.make_inputs(cfg, 1, bias_scale=0.5)
    got = {}
    for gather in ("0", "1"):
        monkeypatch.setenv("KLEOS_GATHER", gather)
        got[gather] = hz.run_layer_single_gpu(cfg, packed[0], forwards=2)
    assert np.array_equal(got["0"][0], got["1"][0]) and np.array_equal(got["0"][1], got["1"][1])
