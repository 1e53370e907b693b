"""The calls whose speed counts: what a program that runs on this package spends its time in.

Four kinds of call, each through the entry point such a program uses:

  ffn       one gated FFN, ``SparseFlowFusedMLP``: built from the three ``nn.Linear`` of a model (``mode`` "auto": the shape gate
            decides per GEMM), or rebuilt from packed weights (``mode`` "packed": ``from_compressed_state``, the form that holds
            no dense copy, so every GEMM is sparse whatever the token count);
  linear    one projection, ``SparseFlowLinear`` with the default policy, with or without bias;
  mlp       ``SparseFlowMLP`` with biases on gate and up (two sparse GEMMs, SiLU.mul, sparse down projection);
  compress  a weight on its way into the package: ``compress_weight`` (dense weight -> values + metadata), ``gate_up`` (the two
            weights of a gated FFN -> one interleaved compressed weight), ``prune`` (the pruned dense copy, any width that is a
            multiple of four) and ``convert`` (prune, check, compress, pack: how a checkpoint is converted).

Weights are N(0, 0.02) and activations N(0, 1), in the 16-bit type of the case, made on the GPU from the seed.
"""
import math

import torch
import torch.nn as nn

from sparseflow_b200 import core, ops
from sparseflow_b200.fused_mlp import SparseFlowFusedMLP
from sparseflow_b200.nn import SparseFlowLinear, SparseFlowMLP, prune_24_dense_weight

_TYPES = {"bf16": torch.bfloat16, "f16": torch.float16}

# Range of the drawn cases.  The largest listed case (8192 x 28672 FFN, 2048 tokens) bounds their cost.
_MOST_FFN = 3 * 2048 * 8192 * 28672
_MOST_WEIGHT = 8192 * 28672


def listed():
    return [
        # generation for one user: one token through the FFN of the headline configuration
        {"name": "ffn_decode_1", "kind": "ffn", "mode": "auto", "hidden": 4096, "inter": 11008, "batch": 1, "seq": 1, "dtype": "bf16", "bias": False},
        # generation for a batch of users, one token each
        {"name": "ffn_decode_24", "kind": "ffn", "mode": "auto", "hidden": 4096, "inter": 14336, "batch": 24, "seq": 1, "dtype": "bf16", "bias": False},
        # a large decode batch on packed weights, ragged
        {"name": "ffn_batch_150", "kind": "ffn", "mode": "packed", "hidden": 4096, "inter": 11008, "batch": 150, "seq": 1, "dtype": "f16", "bias": False},
        # a short prompt / prefill chunk on packed weights, ragged, with a bias
        {"name": "ffn_chunk_300", "kind": "ffn", "mode": "packed", "hidden": 4096, "inter": 11008, "batch": 1, "seq": 300, "dtype": "bf16", "bias": True},
        # a prefill chunk of the usual size of chunked prefill
        {"name": "ffn_chunk_512", "kind": "ffn", "mode": "auto", "hidden": 4096, "inter": 14336, "batch": 1, "seq": 512, "dtype": "bf16", "bias": False},
        # prefill of two sequences: the headline configuration
        {"name": "ffn_prefill_4096", "kind": "ffn", "mode": "auto", "hidden": 4096, "inter": 11008, "batch": 2, "seq": 2048, "dtype": "bf16", "bias": False},
        # prefill on the largest FFN
        {"name": "ffn_prefill_large", "kind": "ffn", "mode": "packed", "hidden": 8192, "inter": 28672, "batch": 1, "seq": 2048, "dtype": "bf16", "bias": False},
        # the smallest call: one token through a small projection with a bias; launch and latency
        {"name": "linear_small_1", "kind": "linear", "op": "o_proj", "rows": 2048, "K": 2048, "batch": 1, "seq": 1, "dtype": "f16", "bias": True},
        # attention projection of a ragged prompt
        {"name": "linear_prompt_1500", "kind": "linear", "op": "q_proj", "rows": 4096, "K": 4096, "batch": 1, "seq": 1500, "dtype": "f16", "bias": False},
        # a gated MLP with biases, the unfused path
        {"name": "mlp_bias_777", "kind": "mlp", "hidden": 4096, "inter": 11008, "batch": 1, "seq": 777, "dtype": "f16"},
        # loading: the two weights of a gated FFN compressed into the fused form
        {"name": "compress_gate_up", "kind": "compress", "form": "gate_up", "rows": 11008, "K": 4096, "dtype": "bf16"},
        # converting a checkpoint's weight to a packed one, with the check that it is 2:4
        {"name": "convert_4096", "kind": "compress", "form": "convert", "rows": 4096, "K": 4096, "dtype": "f16"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _step(v, step, lo):
    return max(lo, v // step * step)


def _tokens(rng, most):
    # batch x sequence: single sequences and batches of single tokens as well as both at once
    n = _log(rng, 1, max(1, most))
    shape = rng.choice(("seq", "batch", "both"))
    if shape == "seq":
        return 1, n
    if shape == "batch":
        return n, 1
    b = rng.randint(1, 8)
    return b, max(1, n // b)


def draw(rng):
    kind = rng.choice(("ffn", "ffn", "ffn", "linear", "linear", "mlp", "compress", "compress"))
    dtype = rng.choice(("bf16", "f16"))
    if kind in ("ffn", "mlp"):
        hidden = _step(_log(rng, 1024, 8192), 64, 64)
        inter = _step(int(hidden * rng.uniform(2.0, 4.0)), 64, 64)
        batch, seq = _tokens(rng, min(8192, _MOST_FFN // (3 * hidden * inter)))
        c = {"kind": kind, "hidden": hidden, "inter": inter, "batch": batch, "seq": seq, "dtype": dtype}
        if kind == "ffn":
            c.update(mode=rng.choice(("auto", "packed")), bias=rng.random() < 0.25)
        return c
    if kind == "linear":
        op = rng.choice(("q_proj", "o_proj", "down_proj", "gate_proj"))
        K = _step(_log(rng, 1024, 8192), 64, 64)
        f = {"q_proj": (1.0, 1.0), "o_proj": (1.0, 1.0), "down_proj": (0.25, 0.5), "gate_proj": (2.0, 4.0)}[op]
        rows = _step(int(K * rng.uniform(*f)), 8, 8)
        batch, seq = _tokens(rng, 8192)
        return {"kind": kind, "op": op, "rows": rows, "K": K, "batch": batch, "seq": seq, "dtype": dtype, "bias": rng.random() < 0.5}
    form = rng.choice(("weight", "gate_up", "prune", "convert"))
    n = _log(rng, 1 << 20, _MOST_WEIGHT)     # weight elements
    K = _log(rng, 512, 16384)
    K = _step(K, {"prune": 4, "weight": 16, "gate_up": 16, "convert": 16}[form], 64)
    rows = _step(max(16, min(n, _MOST_WEIGHT) // K), 16, 16) + (rng.randint(0, 15) if form != "gate_up" else 0)
    return {"kind": kind, "form": form, "rows": rows, "K": K, "dtype": dtype}


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _weight(rows, K, dtype, g):
    return (torch.randn(rows, K, generator=g, device="cuda") * 0.02).to(dtype)


def _kept(w):
    """Mask [groups of four, 4]: 2:4 magnitude pruning keeps the two largest magnitudes, the higher index on a tie."""
    a = w.reshape(-1, 4).abs()
    mine, other = a.unsqueeze(2), a.unsqueeze(1)
    later = torch.ones(4, 4, dtype=torch.bool, device=w.device).triu(1)
    beaten = (other > mine) | ((other == mine) & later)
    return beaten.sum(2, dtype=torch.uint8) <= 1


def _pruned(w):
    return torch.where(_kept(w), w.reshape(-1, 4), torch.zeros((), dtype=w.dtype, device=w.device)).reshape(w.shape)


def _inputs(case, seed):
    """Weights, biases and activations of a case."""
    g, dt, kind = _gen(seed), _TYPES[case["dtype"]], case["kind"]
    if kind == "compress":
        n = 2 if case["form"] == "gate_up" else 1
        return {"w": [_weight(case["rows"], case["K"], dt, g) for _ in range(n)]}
    if kind == "linear":
        d = {"w": [_weight(case["rows"], case["K"], dt, g)], "x_width": case["K"]}
        d["b"] = [_weight(1, case["rows"], dt, g).reshape(-1) * 10 if case["bias"] else None]
    else:
        H, I = case["hidden"], case["inter"]
        shapes = ((I, H), (I, H), (H, I))
        biased = (True, True, True) if kind == "mlp" else (False, False, case["bias"])
        # the fused FFN is handed 2:4 weights (it does not prune); the other modules prune what they get
        made = (_weight(r, k, dt, g) for r, k in shapes)
        d = {"w": [_pruned(w) if kind == "ffn" else w for w in made], "x_width": H}
        d["b"] = [_weight(1, r, dt, g).reshape(-1) * 10 if yes else None for (r, _), yes in zip(shapes, biased)]
    d["x"] = torch.randn(case["batch"], case["seq"], d.pop("x_width"), generator=g, device="cuda").to(dt)
    return d


def _linear(w, b):
    m = nn.Linear(w.shape[1], w.shape[0], bias=b is not None, device="meta")
    m.weight = nn.Parameter(w, requires_grad=False)
    if b is not None:
        m.bias = nn.Parameter(b, requires_grad=False)
    return m


def prepare(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    if kind == "compress":
        return {"kind": kind, "form": case["form"], "w": d["w"]}
    if kind == "ffn":
        m = SparseFlowFusedMLP(*(_linear(w, b) for w, b in zip(d["w"], d["b"])), force_mode="auto")
        if case["mode"] == "packed":
            m = SparseFlowFusedMLP.from_compressed_state(m.compressed_state())
    elif kind == "linear":
        m = SparseFlowLinear(d["w"][0], d["b"][0], op_name=case["op"], dense_uses_pruned=True)
    else:
        m = SparseFlowMLP(case["hidden"], case["inter"], *d["w"], *d["b"], dtype=d["x"].dtype, down_mode="sparse")
    return {"kind": kind, "module": m, "x": d["x"]}


def run(state):
    if state["kind"] != "compress":
        return state["module"](state["x"])
    w, form = state["w"], state["form"]
    if form == "prune":
        return prune_24_dense_weight(w[0])
    if form == "convert":
        return core.compress_2_4(core.prune_2_4(w[0]))
    cw = ops.compress_gate_up(*w) if form == "gate_up" else ops.compress_weight(w[0])
    return {"values": cw.values, "meta": cw.meta}


def work(case):
    """Bytes: 16-bit activations and outputs, weights as 2:4 needs them (half the values and a quarter byte pair of indices per four:
    1.125 bytes an element); operations: the products of the kept half."""
    kind = case["kind"]
    if kind == "compress":
        n = case["rows"] * case["K"] * (2 if case["form"] == "gate_up" else 1)
        return {"bytes": n * (4 if case["form"] == "prune" else 3.125), "flops": 0}
    M = case["batch"] * case["seq"]
    if kind == "linear":
        weights, ends, biases = case["rows"] * case["K"], M * (case["rows"] + case["K"]), case["rows"] if case["bias"] else 0
    else:
        H, I = case["hidden"], case["inter"]
        weights, ends = 3 * H * I, 2 * M * H
        biases = H + 2 * I if kind == "mlp" else H if case["bias"] else 0
    return {"bytes": 1.125 * weights + 2 * (ends + biases), "flops": M * weights}


def tolerance(case):
    """Compression moves bits and is exact.  One projection is rounded once, from 32-bit sums: another order of summation moves
    a few results by one unit in the last place.  In an FFN the hidden values are rounded too, and gate and up where the dense branch or
    the unfused path runs: two to three roundings of 2^-9 (bf16) or 2^-12 (f16) each."""
    if case["kind"] == "compress":
        return "exact"
    if case["kind"] == "linear":
        return {"rel": 4e-3 if case["dtype"] == "bf16" else 5e-4}
    return {"rel": 1e-2 if case["dtype"] == "bf16" else 1.5e-3}


def exact(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    if kind == "compress":
        if case["form"] == "convert":
            return None                     # a packed blob: bytes
        if case["form"] == "prune":
            return _pruned(d["w"][0]).double()
        w = d["w"][0]
        if case["form"] == "gate_up":       # blocks of 16 gate rows, then the 16 matching up rows
            g, u = (t.reshape(-1, 16, t.shape[1]) for t in d["w"])
            w = torch.stack((g, u), dim=1).reshape(-1, w.shape[1])
        return {"values": w.reshape(-1, 4)[_kept(w)].reshape(w.shape[0], -1).double(), "meta": None}

    def times(x, i):
        w = d["w"][i] if kind == "ffn" else _pruned(d["w"][i])
        y = x @ w.double().t()
        return y if d["b"][i] is None else y + d["b"][i].double()

    x = d["x"].double()
    if kind == "linear":
        return times(x, 0)
    gate = times(x, 0)
    h = gate * torch.sigmoid(gate)
    del gate
    return times(h * times(x, 1), 2)
