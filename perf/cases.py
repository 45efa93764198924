"""The work whose speed is measured: one MoE layer forward (or one router call) on one GPU.

A program that uses this library initialises a layer from a configuration, keeps its packed
buffers [A | Wg | W1 | W2 | b1 | b2] and [probs | out] on the GPU and calls ``forward_host`` on
them, once per layer and step; a program that may not allocate calls ``route_static`` instead and
gets the routing alone.  The listed cases are the benchmark layers of ``baseline_config`` and the
layers ``bench.py`` and the tests run beside them.  Activations are N(0,1), weights
N(0,1/sqrt(fan_in)), FFN biases N(0,0.1), as ``aristos_b200/synth.py`` draws them for the tests.
"""
import math

import numpy as np
import torch

from aristos_b200 import kleos
from aristos_b200.config import KleosConfig

_DTYPE = {"fp32": 0, "tf32": 1, "bf16": 2, "fp16": 3}
_TORCH = {"fp32": torch.float32, "tf32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}


def _case(name, dtype, S, H, I, E, K=2, cf=1.0, act="relu", drop=True, zipf=0.0, train=False, entry="layer"):
    c = dict(dtype=dtype, S=S, H=H, I=I, E=E, K=K, cf=cf, act=act, drop=drop, zipf=zipf, train=train, entry=entry)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest layer, in the reference's own element type: nothing but latency and launches
        _case("c1_fp32", "fp32", 256, 512, 1024, 8),
        # the same size in bf16: a small model's layer, or a short prompt
        _case("c1_bf16", "bf16", 256, 512, 1024, 8),
        # serving, one step of decode: 128 sequences, no token dropped, every expert's weights read
        _case("decode_bf16", "bf16", 128, 2048, 2048, 64, drop=False),
        # the float layer in the reference's element type, and its TF32 form
        _case("c2_fp32", "fp32", 4096, 2048, 2048, 16),
        _case("c2_tf32", "tf32", 4096, 2048, 2048, 16),
        # prefill of the layer that the headline metric is quoted on
        _case("c3_bf16", "bf16", 8192, 2048, 2048, 64),
        # a hot-expert layer: Zipf popularity, full cells and dropped tokens, two gate column tiles
        _case("c4_zipf_bf16", "bf16", 16384, 2048, 2048, 128, cf=1.25, zipf=1.2),
        # the large FFN: the tensor pipe's own speed
        _case("c5_bf16", "bf16", 4096, 4096, 14336, 8),
        # ragged: fp16, GELU, odd panel counts, an intermediate size that ends inside a tile, top-4
        _case("ragged_fp16_gelu", "fp16", 2944, 1088, 2880, 24, K=4, cf=1.25, act="gelu"),
        # training: the forward with the gate statistics, whose loss the program reads each step
        _case("train_bf16", "bf16", 4096, 2048, 2048, 32, train=True),
        # num_experts = 1: the dense FFN
        _case("dense_bf16", "bf16", 4096, 2048, 2048, 1, K=1),
        # the router alone, without an allocation, for a program that runs its own experts
        _case("route_static_bf16", "bf16", 4096, 2048, 0, 64, entry="route_static"),
    ]


def _log(rng, lo, hi, step):
    """A multiple of `step` between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def _pick(rng):
    kind = rng.choice(["layer"] * 6 + ["dense", "train", "route_static", "decode"])
    if kind == "route_static":
        E = rng.choice([8, 16, 24, 48, 64])
        return _case(None, rng.choice(["bf16", "bf16", "fp32"]), _log(rng, 128, 4096, 32), _log(rng, 512, 4096, 64), 0, E,
                     K=rng.choice([1, 2, 2, 4, 8]), entry=kind)
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16", "fp32", "tf32"])
    S, H, I = _log(rng, 256, 16384, 128), _log(rng, 512, 4096, 64), _log(rng, 1024, 14336, 64)
    act = rng.choice(["relu", "relu", "gelu"])
    if kind == "dense":
        return _case(None, dtype, S, H, I, 1, K=1, act=act)
    E = rng.choice([8, 12, 16, 24, 32, 64, 128])
    if kind == "decode":
        return _case(None, rng.choice(["bf16", "fp16"]), rng.choice([128, 256]), H, I, E, K=2, act=act, drop=False)
    return _case(None, dtype, S, H, I, E, K=rng.choice([1, 2, 2, 2, 4]), cf=rng.choice([1.0, 1.0, 1.25, 2.0]), act=act,
                 zipf=rng.choice([0.0, 0.0, 0.0, 1.2]), train=kind == "train")


def draw(rng):
    # no dearer than the dearest listed case of its kind: the large FFN's arithmetic (the float
    # layer's for 32-bit elements) and the hot-expert layer's weights
    while True:
        c = _pick(rng)
        flops = 4.0 * c["S"] * c["K"] * c["H"] * c["I"]
        weights = 2.0 * c["E"] * c["H"] * c["I"]
        if flops <= (1.9e12 if c["dtype"] in ("bf16", "fp16") else 1.37e11) and weights <= 1.1e9:
            return c


# ---------------------------------------------------------------------------- inputs
def _config(case):
    return KleosConfig(sequence_len=case["S"], hidden_size=case["H"], intermediate_size=case["I"], num_experts=case["E"],
                       expert_top_k=case["K"], capacity_factor=case["cf"], drop_tokens=int(case["drop"]),
                       hidden_act=int(case["act"] == "gelu"), is_training=int(case["train"]), torch_dtype=_DTYPE[case["dtype"]])


def _round(x, dtype):
    """fp32 values as elements of the layer, in the storage the library expects."""
    if dtype == "tf32":  # an fp32 word with a 10-bit mantissa
        u = x.view(torch.int32)
        return ((u + 0xFFF + ((u >> 13) & 1)) & -8192).view(torch.float32)
    return x.to(_TORCH[dtype])


def _sections(case):
    """Names, sizes and standard deviations of the packed input, in order."""
    S, H, I, E = case["S"], case["H"], case["I"], case["E"]
    px = -(-E // 64) * 64
    gate = [("Wg", E * H, H ** -0.5), ("pad", (px - E) * H, 0.0)] if E > 1 else []
    ffn = [("W1", E * I * H, H ** -0.5), ("W2", E * H * I, I ** -0.5 if I else 0.0), ("b1", E * I, 0.1), ("b2", E * H, 0.1)]
    return [("A", S * H, 1.0)] + gate + (ffn if case["entry"] == "layer" or I else [])


def _inputs(case, seed):
    """The packed input on the GPU, and where each section starts."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    parts = _sections(case)
    packed = torch.empty(sum(n for _, n, _ in parts), dtype=_TORCH[case["dtype"]], device="cuda")
    at, start = 0, {}
    for name, n, std in parts:
        start[name] = at
        for i in range(at, at + n, 1 << 26):
            m = min(1 << 26, at + n - i)
            x = torch.randn(m, generator=gen, device="cuda").mul_(std) if std else torch.zeros(m, device="cuda")
            packed[i:i + m] = _round(x, case["dtype"])
        at += n
    return packed, start


def _gate_bias(case):
    """Logit bias that makes expert popularity follow Zipf over a fixed permutation; it belongs to
    the layer, as its configuration does, and not to one step's inputs."""
    rank = np.random.RandomState(case["E"]).permutation(case["E"]) + 1.0
    pmf = rank ** -case["zipf"]
    return np.log(pmf / pmf.sum()).astype(np.float32)


_layer = None  # configuration of the layer this process has initialised (the library holds one at a time)


def _ensure_layer(case):
    global _layer
    key = {k: v for k, v in case.items() if k != "name"}
    if _layer == key:
        return
    if _layer is not None:
        kleos.finalize()
        _layer = None
    kleos.initialize(_config(case))
    _layer = key
    if case["zipf"]:
        kleos.set_gate_bias(_gate_bias(case))


def prepare(case, seed):
    if case["entry"] != "route_static":
        _ensure_layer(case)
    packed, start = _inputs(case, seed)
    S, H, E, K = case["S"], case["H"], case["E"], case["K"]
    px = -(-E // 64) * 64 if E > 1 else 0
    if case["entry"] == "route_static":
        dev = dict(device="cuda")
        return dict(case=case, packed=packed, A=packed[:S * H], Wg=packed[start["Wg"]:],
                    probs=torch.empty(S, px, dtype=packed.dtype, **dev), topk=torch.empty(S, K, dtype=torch.int32, **dev),
                    mcw=torch.empty(S, dtype=torch.float32, **dev))
    result = torch.empty(S * px + S * H, dtype=packed.dtype, device="cuda")
    outputs = dict(out=result[S * px:].view(S, H))
    if px:
        outputs["probs"] = result[:S * px].view(S, px)
    return dict(case=case, packed=packed, result=result, outputs=outputs,
                info=kleos.get_info() if case["train"] else None)


def run(state):
    case = state["case"]
    stream = torch.cuda.current_stream().cuda_stream or None
    if case["entry"] == "route_static":
        kleos.route_static(state["A"], state["Wg"], None, case["S"], case["H"], case["E"], case["K"], _DTYPE[case["dtype"]],
                           state["probs"], state["topk"], state["mcw"], stream)
        return dict(probs=state["probs"], topk=state["topk"], mcw=state["mcw"])
    kleos.forward_host(state["packed"], state["result"], stream)
    if case["train"]:  # the loss is read on the host, as a training step does
        return dict(state["outputs"], **kleos.gate_stats(state["info"]))
    return state["outputs"]


# ---------------------------------------------------------------------------- what a pass has to do
def _capacity(case):
    base = -(-case["S"] // case["E"]) if case["drop"] else case["S"]
    return int(math.ceil(base * case["cf"] - 1e-9)) * case["K"]


def _expected_rows(case):
    """Rows each expert is expected to process: the gate's logits are N(0,1) plus the bias."""
    logits = np.random.RandomState(1).standard_normal((2048, case["E"]))
    if case["zipf"]:
        logits = logits + _gate_bias(case)
    top = np.argpartition(-logits, case["K"] - 1, axis=1)[:, :case["K"]]
    n = np.bincount(top.ravel(), minlength=case["E"]) * (case["S"] / 2048.0)
    return np.minimum(n, _capacity(case))


def work(case):
    S, H, I, E, K = case["S"], case["H"], case["I"], case["E"], case["K"]
    size = 2 if case["dtype"] in ("bf16", "fp16") else 4
    if E == 1:
        return dict(bytes=size * (2.0 * S * H + 2.0 * H * I + H + I), flops=4.0 * S * H * I)
    px = -(-E // 64) * 64
    if case["entry"] == "route_static":
        return dict(bytes=size * (S * H + E * H + S * px) + 4.0 * S * (K + 1), flops=2.0 * S * H * E)
    rows = _expected_rows(case)
    used = float(np.minimum(rows, 1.0).sum())  # experts whose weights are needed at all
    return dict(bytes=size * (2.0 * S * H + E * H + S * px + used * (2.0 * H * I + H + I)),
                flops=2.0 * S * H * E + 4.0 * float(rows.sum()) * H * I)


def tolerance(case):
    # About four times the difference between this path and exact() below, which rounds nothing:
    # 32-bit sums; TF32 and fp16 keep a 10-bit mantissa, bf16 a 7-bit one, of the gate probabilities,
    # the intermediate, the second GEMM's rows and each step of the combine.
    rel = {"fp32": 1e-5, "tf32": 2e-3, "fp16": 2e-3, "bf16": 1.2e-2}[case["dtype"]]
    if case["entry"] == "route_static":
        return {"rel": rel, "differ": 2e-3}  # two chosen experts with equal 32-bit logits, in either order
    return {"rel": rel}


# ---------------------------------------------------------------------------- 64-bit results
def _act(z, act):
    return torch.relu_(z) if act == "relu" else 0.5 * z * (1.0 + torch.erf(z / math.sqrt(2.0)))


def exact(case, seed):
    packed, at = _inputs(case, seed)
    S, H, I, E, K = case["S"], case["H"], case["I"], case["E"], case["K"]

    def part(name, shape, offset=0):
        n = int(np.prod(shape))
        return packed[at[name] + offset:at[name] + offset + n].view(shape).double()

    A = part("A", (S, H))
    if E == 1:
        y = _act(A @ part("W1", (I, H)).T + part("b1", (I,)), case["act"])
        return dict(out=y @ part("W2", (H, I)).T + part("b2", (H,)))
    logits = A @ part("Wg", (E, H)).T
    if case["zipf"]:
        logits = logits + torch.from_numpy(_gate_bias(case)).cuda().double()
    p = torch.softmax(logits, 1)
    top = torch.sort(logits, dim=1, descending=True, stable=True).indices[:, :K]
    mcw = p.gather(1, top).sum(1)
    probs = torch.zeros(S, -(-E // 64) * 64, dtype=torch.float64, device="cuda")
    probs[:, :E] = p
    if case["entry"] == "route_static":
        return dict(probs=probs, topk=top.int(), mcw=mcw)
    chosen = torch.zeros(S, E, dtype=torch.int32, device="cuda").scatter_(1, top, 1)
    slot = torch.cumsum(chosen, 0) - 1
    out = torch.zeros(S, H, dtype=torch.float64, device="cuda")
    for e in range(E):
        t = torch.nonzero((chosen[:, e] > 0) & (slot[:, e] < _capacity(case))).view(-1)
        if t.numel() == 0:
            continue
        y = _act(A[t] @ part("W1", (I, H), e * I * H).T + part("b1", (I,), e * I), case["act"])
        y = y @ part("W2", (H, I), e * H * I).T + part("b2", (H,), e * H)
        out[t] += y * (p[t, e] / mcw[t])[:, None] if K > 1 else y
    got = dict(out=out, probs=probs)
    if case["train"]:
        mean_prob, mean_count = p.mean(0), chosen.double().mean(0)
        got.update(mean_prob=mean_prob, mean_count=mean_count, loss=float((mean_prob * mean_count).sum() / E))
    return got
