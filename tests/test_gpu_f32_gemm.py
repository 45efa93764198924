"""Float layers: the split-operand tensor-core GEMM at the edges of its tiles, and on operands whose
sums are not finite, where it has to give what fp32 multiply-adds give."""
import numpy as np
import pytest

from aristos_b200 import synth
from aristos_b200.config import KleosConfig
from oracle import c_oracle, moe_oracle
from tests import moe_harness as hz

pytestmark = pytest.mark.gpu


def _cfg(**kw):
    return KleosConfig(**{**dict(sequence_len=256, hidden_size=512, intermediate_size=1024, num_experts=8, torch_dtype=0), **kw})


@pytest.mark.parametrize("kw", [
    dict(sequence_len=128, hidden_size=64, intermediate_size=64, num_experts=4),       # one tile, two K slices
    dict(sequence_len=384, hidden_size=192, intermediate_size=320, num_experts=2),     # odd panel count, 64-column tail
    dict(sequence_len=2048, hidden_size=256, intermediate_size=2112, num_experts=2, hidden_act=1),  # wide tiles, tail, GELU
    dict(sequence_len=1024, hidden_size=704, intermediate_size=448, num_experts=64),   # more experts than block pairs / 2
], ids=["smallest", "odd-panels", "wide-tail-gelu", "many-experts"])
def test_tile_edges(kw):
    cfg = _cfg(**kw)
    packed, views = hz.make_inputs(cfg, 1, bias_scale=0.5)
    ref = moe_oracle.moe_forward(cfg, 1, views)[0]
    probs, out, routing = hz.run_layer_single_gpu(cfg, packed[0], forwards=2)
    hz.check_against_oracle(cfg, ref, probs, out, routing)


def test_operands_of_very_different_size():
    """Rows scaled by 1e-30 .. 1e30: relative accuracy does not depend on a row's size."""
    cfg = _cfg(num_experts=1, expert_top_k=1)
    packed, views = hz.make_inputs(cfg, 1)
    scale = np.float32(10.0) ** np.linspace(-30, 30, cfg.S).astype(np.float32)
    a = packed[0][:cfg.S * cfg.H].reshape(cfg.S, cfg.H)
    a *= scale[:, None]
    ref = c_oracle.dense_ffn(cfg, synth.split_packed(cfg, packed[0], 1))
    _, out, _ = hz.run_layer_single_gpu(cfg, packed[0])
    err = np.abs(out - ref).max(axis=1) / np.abs(ref).max(axis=1)
    assert err.max() <= hz.TOL[0]


@pytest.mark.parametrize("act", [0, 1], ids=["relu", "gelu"])
def test_values_that_are_not_finite(monkeypatch, act):
    """Infinities, NaN and sums that overflow: the same values as from the FP32 FMA kernel."""
    cfg = _cfg(num_experts=1, expert_top_k=1, hidden_act=act)
    packed, _ = hz.make_inputs(cfg, 1, bias_scale=0.5)
    a = packed[0][:cfg.S * cfg.H].reshape(cfg.S, cfg.H)
    a[3, 5], a[40, 511], a[70, 0] = np.inf, -np.inf, np.nan
    a[130] *= np.float32(1e38)
    a[200, :4] = np.float32(3.4e38)
    got = hz.run_layer_single_gpu(cfg, packed[0])[1]
    monkeypatch.setenv("KLEOS_DEBUG_SIMT_GEMM", "1")
    want = hz.run_layer_single_gpu(cfg, packed[0])[1]
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
    assert not np.isfinite(want[[3, 40, 70]]).all()
    plain = np.ones(cfg.S, bool)
    plain[[3, 40, 70, 130, 200]] = False
    # two fp32 results, each within the layer's bound of the 64-bit one
    assert np.abs(got[plain] - want[plain]).max() <= 2 * hz.TOL[0] * np.abs(want[plain]).max()


# tile widths of both GEMMs: 64 columns (one round of tiles either way) and 128 (half as many rounds)
WIDTHS = pytest.mark.parametrize("S,N", [(256, 512), (2048, 2048)], ids=["narrow", "wide"])


@WIDTHS
def test_rows_of_a_single_term(S, N):
    """One nonzero activation in a row: every sum is one product, as exact as a rounded fp32 product.
    Of the product's nine part products the trailing times the trailing one is left out (under 2^-30 of
    the product), the sum of the small ones is cut off below 2^-28, and the result is rounded once."""
    rng = np.random.default_rng(S)
    A = np.zeros((S, N), np.float32)
    k = rng.integers(0, N, S)
    A[np.arange(S), k] = (1 + rng.random(S)) * np.exp2(rng.integers(-20, 20, S))
    W1 = (1 + rng.random((N, N))).astype(np.float32)
    A[0, k[0]] = W1[0, k[0]] = np.float32(1 + 2.0 ** -7 - 2.0 ** -23)  # long middle and trailing parts
    zeros = np.zeros(N, np.float32)
    packed = np.concatenate([A.ravel(), W1.ravel(), np.eye(N, dtype=np.float32).ravel(), zeros, zeros])
    cfg = _cfg(sequence_len=S, hidden_size=N, intermediate_size=N, num_experts=1, expert_top_k=1)
    out = hz.run_layer_single_gpu(cfg, packed)[1]
    want = A.sum(1, dtype=np.float64)[:, None] * W1.T.astype(np.float64)[k]
    assert (np.abs(out - want) / want).max() <= 2.0 ** -24 * (1 + 2.0 ** -4)


@WIDTHS
def test_a_token_that_is_not_finite_leaves_the_others(S, N):
    """The other tokens' results are the same bits with and without it."""
    cfg = _cfg(sequence_len=S, hidden_size=N, intermediate_size=N, num_experts=1, expert_top_k=1, hidden_act=1)
    packed, _ = hz.make_inputs(cfg, 1, bias_scale=0.5)
    plain = hz.run_layer_single_gpu(cfg, packed[0])[1]
    a = packed[0][:S * N].reshape(S, N)
    a[5, 7], a[40, N - 1], a[S - 1, 0] = np.nan, np.inf, -np.inf
    got = hz.run_layer_single_gpu(cfg, packed[0])[1]
    hit = [5, 40, S - 1]
    assert not np.isfinite(got[hit]).any()
    assert np.array_equal(np.delete(got, hit, 0), np.delete(plain, hit, 0))


@pytest.mark.parametrize("kw", [dict(), dict(sequence_len=4096, hidden_size=1024, intermediate_size=2048, num_experts=4)],
                         ids=["narrow", "wide"])
def test_expert_weights_that_are_not_finite(monkeypatch, kw):
    """Infinities and NaN in a routed layer's weights: the same values as from the FP32 FMA kernel, the
    experts beside them bit for bit as without."""
    cfg = _cfg(drop_tokens=0, **kw)
    packed, views = hz.make_inputs(cfg, 1, bias_scale=0.5)
    plain = hz.run_layer_single_gpu(cfg, packed[0])[1]
    v = synth.split_packed(cfg, packed[0], 1)
    v["W1"][1, 3, 5], v["W2"][2, 9, 70], v["W2"][2, 11, 71], v["W1"][2, 0, 0] = np.inf, -np.inf, np.nan, np.float32(3.4e38)
    assert not np.isfinite(packed[0]).all()
    _, got, routing = hz.run_layer_single_gpu(cfg, packed[0])
    monkeypatch.setenv("KLEOS_DEBUG_SIMT_GEMM", "1")
    want = hz.run_layer_single_gpu(cfg, packed[0])[1]
    for same in (np.isnan, np.isposinf, np.isneginf):
        assert np.array_equal(same(got), same(want)) and same(want).any()
    untouched = ~np.isin(routing["topk"], [1, 2]).any(1)
    assert untouched.any() and np.array_equal(got[untouched], plain[untouched])


@WIDTHS
def test_dense_result_at_any_float(S, N):
    """The result of a dense float layer may lie at any address that a float may have."""
    import torch
    from aristos_b200 import kleos
    cfg = _cfg(sequence_len=S, hidden_size=N, intermediate_size=N, num_experts=1, expert_top_k=1)
    iP = torch.from_numpy(hz.make_inputs(cfg, 1, bias_scale=0.5)[0][0]).cuda()
    kleos.initialize(cfg, 0, 1)
    try:
        results = []
        for offset in (0, 1, 2, 3):
            buf = torch.full((S * N + 8,), 7.0, device="cuda")
            kleos.forward_host(iP, buf.data_ptr() + 4 * offset)
            assert kleos.last_status().code == 0
            assert (buf[:offset] == 7).all() and (buf[offset + S * N:] == 7).all()
            results.append(buf[offset:offset + S * N].clone())
    finally:
        kleos.finalize()
    assert all(torch.equal(r, results[0]) for r in results) and not (results[0] == 7).any()
