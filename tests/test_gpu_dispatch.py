"""One rank's dispatch and panel list (token by token, written by the router) against the kernels that
several ranks use (dispatch_kernel, plan_kernel), which KLEOS_DISPATCH_KERNELS=1 runs on one rank too."""
import numpy as np
import pytest

from aristos_b200.config import KleosConfig
from oracle import moe_oracle
from tests import moe_harness as hz

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [
    dict(num_experts=2, expert_top_k=1),
    dict(num_experts=3),
    dict(num_experts=31, expert_top_k=8),                                   # dropped tokens
    dict(num_experts=32, drop_tokens=0),
    dict(num_experts=33, sequence_len=384, expert_top_k=4),                # one more than a warp scans at a time
    dict(num_experts=64, sequence_len=1024, capacity_factor=1.25),
    dict(num_experts=96, sequence_len=1152, expert_top_k=3, is_training=1),
    dict(num_experts=128, sequence_len=2048),
    dict(num_experts=256, sequence_len=512, expert_top_k=4),
], ids=lambda kw: "-".join(str(v) for v in kw.values()))
@pytest.mark.parametrize("dtype", [0, 1, 2])
@pytest.mark.parametrize("empty", [False, True], ids=["", "empty-experts"])
def test_same_bits_as_the_kernels_of_several_ranks(monkeypatch, dtype, kw, empty):
    cfg = KleosConfig(**{**dict(sequence_len=256, hidden_size=192, intermediate_size=128, torch_dtype=dtype), **kw})
    packed, views = hz.make_inputs(cfg, 1, bias_scale=0.5)
    bias = None
    if empty:  # every third expert gets no token, the first and the last among them where k experts remain
        bias = np.where(np.arange(cfg.E) % 3 == 0, -100.0, 0.0).astype(np.float32)
        bias[-1] = -100.0
        if (bias == 0).sum() < cfg.K:
            pytest.skip("too few experts remain")
    ref = moe_oracle.moe_forward(cfg, 1, views, bias)[0]
    runs = []
    for kernels in ("0", "1"):
        monkeypatch.setenv("KLEOS_DISPATCH_KERNELS", kernels)
        probs, out, routing = hz.run_layer_single_gpu(cfg, packed[0], gate_bias=bias, forwards=2)
        hz.check_against_oracle(cfg, ref, probs, out, routing)
        runs.append(dict(routing, probs=probs, out=out))
    assert not empty or (runs[0]["counts"] == 0).any()
    for name in runs[0]:
        assert np.array_equal(runs[0][name], runs[1][name]), name
