"""kleos_route_static on bf16 when a wait runs out: the first of a cluster's four blocks withholds its partial
logits, the other three give up after KLEOS_WAIT_MS, their tokens say so, and the context goes on."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import torch
from aristos_b200 import kleos
S, H, E, K = 300, 512, 16, 2
g = torch.Generator(device="cuda").manual_seed(3)
A = torch.randn(S, H, generator=g, device="cuda").bfloat16()
Wg = torch.zeros(64, H, dtype=torch.bfloat16, device="cuda")
Wg[:E] = torch.randn(E, H, generator=g, device="cuda").bfloat16()
probs = torch.zeros(S, 64, dtype=torch.bfloat16, device="cuda")
topk, mcw = torch.full((S, K), 5, dtype=torch.int32, device="cuda"), torch.full((S,), 0.5, device="cuda")
kleos.route_static(A, Wg, None, S, H, E, K, 2, probs, topk, mcw)
torch.cuda.synchronize()
first = torch.arange(S, device="cuda") % 128 < 32   # the withholding block has the others' parts
want = torch.topk(A.double() @ Wg[:E].double().T, K, dim=1).indices
assert torch.equal(topk[first].sort(1).values, want[first].int().sort(1).values)
assert torch.isfinite(mcw[first]).all()
assert (topk[~first] == -1).all() and torch.isnan(mcw[~first]).all()
print("told")
"""


def test_a_wait_that_runs_out_is_told():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, KLEOS_WAIT_MS="50", KLEOS_DEBUG_STATIC_WITHHOLD="1", PYTHONPATH=root)
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, cwd=root, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "told" in r.stdout, r.stderr[-2000:]
