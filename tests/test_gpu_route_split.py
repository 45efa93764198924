"""The one-launch router of 16-bit and TF32 layers: one, two and four blocks per 128 tokens, K parts of one
slice, more blocks of tokens than the chip holds at once, every width of the selection, and exact ties."""
import numpy as np
import pytest

from aristos_b200.config import KleosConfig
from oracle import moe_oracle
from tests import moe_harness as hz

pytestmark = pytest.mark.gpu


def _cfg(S, H, E, K, dtype, **kw):
    return KleosConfig(sequence_len=S, hidden_size=H, intermediate_size=64, num_experts=E, expert_top_k=K, torch_dtype=dtype, **kw)


@pytest.mark.parametrize("S,H,E,K,dtype", [
    (128, 64, 3, 2, 2),       # a single slice of K: one block per 128 tokens
    (128, 64, 3, 2, 1),       # ... two slices: two blocks
    (128, 192, 64, 8, 3),     # three slices: two blocks
    (384, 320, 33, 1, 2),     # parts of unequal length
    (256, 256, 65, 4, 2),     # 128 columns
    (4864, 128, 64, 2, 2),    # 38 times 4 blocks do not fit: two
    (9600, 128, 17, 3, 1),    # 75 times 2 do not: one
    (19200, 64, 128, 2, 2),   # 150 blocks of 128 tokens: a second round for some
], ids=lambda v: str(v))
def test_parts_and_rounds(S, H, E, K, dtype):
    cfg = _cfg(S, H, E, K, dtype)
    packed, views = hz.make_inputs(cfg, 1, bias_scale=0.5)
    ref = moe_oracle.moe_forward(cfg, 1, views)[0]
    probs, out, routing = hz.run_layer_single_gpu(cfg, packed[0], forwards=3)
    hz.check_against_oracle(cfg, ref, probs, out, routing)


@pytest.mark.parametrize("E,K", [(64, 2), (100, 5)])
def test_exact_ties_go_to_the_lowest_id(E, K):
    """Tokens of zeros have equal logits for all experts: every one of them is re-evaluated, and the first k win."""
    cfg = _cfg(256, 128, E, K, 2, drop_tokens=0)
    packed, views = hz.make_inputs(cfg, 1)
    views[0]["A"][::3] = 0.0
    _, _, routing = hz.run_layer_single_gpu(cfg, packed[0], forwards=2)
    assert (np.sort(routing["topk"][::3], axis=1) == np.arange(K)).all()


def test_tokens_that_are_not_finite_leave_the_others_slots():
    """A token of NaN logits chooses expert 0 k times over; counts and slots of the finite tokens do not move."""
    S, E, K = 384, 64, 8
    cfg = _cfg(S, 128, E, K, 2, drop_tokens=0)
    packed, views = hz.make_inputs(cfg, 1)
    finite = np.ones(S, bool)
    finite[40:160] = False
    ref = moe_oracle.moe_forward(cfg, 1, views)[0]
    views[0]["A"][~finite] = np.nan
    _, out, routing = hz.run_layer_single_gpu(cfg, packed[0], forwards=2)
    assert np.array_equal(np.sort(routing["topk"][finite], 1), np.sort(ref["topk"][finite], 1))
    assert (routing["topk"][~finite] == 0).all()
    chosen = routing["topk"].ravel()
    assert np.array_equal(routing["counts"], np.bincount(chosen, minlength=E))
    slots = routing["slots"].ravel()
    for e in range(E):  # ascending token order
        assert np.array_equal(slots[chosen == e], np.arange((chosen == e).sum()))
    want = ref["out"][finite]
    assert np.abs(out[finite] - want).max() <= hz.TOL[2] * np.abs(want).max()
