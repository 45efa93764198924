"""16-bit layers: a token's probabilities and mCw do not depend on how many other tokens the layer has: however the router spreads
the tokens over the chip (32, 64 or 128 a block), every logit is one sum over all of K, and the softmax sum goes by experts."""
import numpy as np
import pytest

from aristos_b200.config import KleosConfig
from tests import moe_harness as hz

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,E,K,train", [(2, 64, 2, 0), (2, 24, 4, 0), (3, 128, 2, 1)], ids=["bf16", "bf16-top4", "fp16-training"])
def test_same_bits_at_every_size(dtype, E, K, train):
    got = []
    for S in (128, 4864, 9600):
        cfg = KleosConfig(sequence_len=S, hidden_size=1024, intermediate_size=64, num_experts=E, expert_top_k=K, torch_dtype=dtype, is_training=train)
        packed, views = hz.make_inputs(cfg, 1)
        if got:
            views[0]["A"][-128:] = got[0][2]
        probs, _, routing = hz.run_layer_single_gpu(cfg, packed[0])
        got.append((probs[-128:], routing["mcw"][-128:], views[0]["A"][-128:].copy()))
    for probs, mcw, _ in got[1:]:
        assert np.array_equal(probs, got[0][0]) and np.array_equal(mcw, got[0][1])
