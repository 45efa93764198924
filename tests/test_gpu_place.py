"""Slots by place_kernel with 32, 64 and 128 tokens a block, and top-8, where a block of 128 has more choices than
threads; a capacity that drops rows, so that every slot counts."""
import numpy as np
import pytest

from aristos_b200 import synth
from aristos_b200.config import KleosConfig
from oracle import moe_oracle
from tests import moe_harness as hz

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,E,K,dtype,train", [(18944, 4, 1, 0, 0), (18944 + 128, 8, 8, 0, 0), (37888 + 128, 130, 2, 2, 0), (37888 + 384, 8, 8, 0, 1)],
                         ids=["32", "64", "128-wide", "128-top8-training"])
def test_tokens_a_block(S, E, K, dtype, train):
    cfg = KleosConfig(sequence_len=S, hidden_size=64, intermediate_size=64, num_experts=E, expert_top_k=K, torch_dtype=dtype,
                      is_training=train)
    packed, views = hz.make_inputs(cfg, 1)
    ref = moe_oracle.route(cfg, views[0]["A"], views[0]["Wg"])
    _, _, routing = hz.run_layer_single_gpu(cfg, packed[0], forwards=2)
    assert np.array_equal(routing["counts"], ref["counts"])

    def by_expert(r):
        m = np.full((S, E), -2, np.int64)
        np.put_along_axis(m, r["topk"].astype(np.int64), r["slots"].astype(np.int64), 1)
        return m

    assert np.array_equal(by_expert(routing), by_expert(ref))
