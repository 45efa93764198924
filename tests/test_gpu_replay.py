"""A captured forward, replayed on other tokens: every replay carries the same kernel arguments (the epoch among
them), so nothing that a forward leaves on the GPU may pass for the next one's."""
import pytest

from aristos_b200 import kleos, synth
from aristos_b200.config import KleosConfig
from tests import moe_harness as hz

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,E,dtype,kw", [
    (256, 8, 2, {}),                      # rows gathered
    (4096, 64, 2, {}),                    # several blocks per 128 tokens
    (4096, 8, 3, dict(is_training=1)),    # rows copied
    (2048, 16, 1, {}),
    (2048, 16, 0, {}),                    # place_kernel
    (2048, 200, 2, {}),                   # ... behind the router of more than 128 experts
    (19200, 16, 2, {}),                   # a second round of blocks
], ids=lambda v: str(v))
def test_replays_follow_their_tokens(S, E, dtype, kw):
    import torch
    cfg = KleosConfig(sequence_len=S, hidden_size=128, intermediate_size=128, num_experts=E, expert_top_k=2, torch_dtype=dtype, **kw)
    raw = torch.from_numpy(synth.encode(hz.make_inputs(cfg, 1)[0][0], dtype)).cuda()
    n = cfg.S * cfg.H
    tokens = [torch.from_numpy(synth.encode(synth.round_to_dtype(synth.activations(cfg, 0, 77 + i).ravel(), dtype), dtype)).cuda()
              for i in range(3)]
    info = kleos.initialize(cfg)
    try:
        out = torch.zeros(info.output_elems, dtype=raw.dtype, device="cuda")
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            want = []
            for t in tokens:
                raw[:n].copy_(t)
                kleos.forward_host(raw, out, stream.cuda_stream)
                want.append(out.clone())
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                kleos.forward_host(raw, out, stream.cuda_stream)
            for i in (1, 0, 2, 0, 1):
                raw[:n].copy_(tokens[i])
                out.zero_()
                graph.replay()
                stream.synchronize()
                assert torch.equal(out, want[i])
            del graph
    finally:
        kleos.finalize()
