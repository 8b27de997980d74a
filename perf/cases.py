"""Performance cases of the W4A16 GEMM: what a program that serves quantised linear layers asks of this package.

A case is one kind of call and its sizes:

* ``gemm``   one layer, eager: ``Layer.forward`` (allocates its output) or ``mul`` into a kept output
* ``step``   the four linear layers of a decoder block (fused qkv, attention output, fused gate-up, down), eager ``mul``
* ``graph``  the same for several blocks, captured once in a CUDA graph and replayed, as a decode loop does
* ``host``   the four layers of a block with activations and results in pinned host memory (``HostGemm``)
* ``pack``   quantise and pack a layer on the device (``quantize_pack_device``), which loading a model does per layer

Layers are those that ``Layer`` accepts: k a multiple of 128, n of 256, group size 128 or one scale per column (-1).
"""
import importlib
import math

import torch

w4 = importlib.import_module("awesome-cute_b200")


def listed():
    return [
        # one token through a narrow layer (the k/v projection of the 70B shapes): start-up, launch and host time only
        {"name": "kv_proj_m1", "kind": "gemm", "call": "layer", "m": 1, "n": 1024, "k": 8192, "group": 128},
        # a few tokens through a layer of no round size, k an odd multiple of 128 (a split of a deeper layer)
        {"name": "odd_layer_m5", "kind": "gemm", "call": "mul", "m": 5, "n": 3328, "k": 4480, "group": 128},
        # the decode step of the 7B shapes at 16 sequences, captured in a graph: the memory-bound regime
        {"name": "decode_graph_m16", "kind": "graph", "m": 16, "hidden": 4096, "ffn": 11008, "blocks": 4, "group": 128},
        # the same block one call after the other with the activations on the host
        {"name": "host_block_m16", "kind": "host", "m": 16, "hidden": 4096, "ffn": 11008, "group": 128},
        # the largest layer of the 70B shapes at a small batch: all weight traffic
        {"name": "gate_up_70b_m8", "kind": "gemm", "call": "mul", "m": 8, "n": 57344, "k": 8192, "group": 128},
        # a batch of 48 sequences, or a short prompt
        {"name": "gate_up_7b_m48", "kind": "gemm", "call": "layer", "m": 48, "n": 22016, "k": 4096, "group": 128},
        # an odd batch on per-channel scales
        {"name": "per_channel_m77", "kind": "gemm", "call": "mul", "m": 77, "n": 5120, "k": 5504, "group": -1},
        # the deepest layer of the 70B shapes at 128 rows: few tiles, long k
        {"name": "down_70b_m128", "kind": "gemm", "call": "mul", "m": 128, "n": 8192, "k": 28672, "group": 128},
        # prefill of a 1024-token prompt through one block of the 7B shapes
        {"name": "prefill_block_m1024", "kind": "step", "m": 1024, "hidden": 4096, "ffn": 11008, "group": 128},
        # prompts of uneven lengths concatenated: a ragged large batch, 13B shapes
        {"name": "prefill_m1537", "kind": "gemm", "call": "layer", "m": 1537, "n": 13824, "k": 5120, "group": 128},
        # the largest call: a 4096-token prompt through the 70B gate-up layer
        {"name": "prefill_70b_m4096", "kind": "gemm", "call": "mul", "m": 4096, "n": 57344, "k": 8192, "group": 128},
        # loading: one fp16 layer quantised and packed
        {"name": "pack_7b_gate_up", "kind": "pack", "n": 22016, "k": 4096, "group": 128},
    ]


def _log(rng, lo, hi, step):
    """A multiple of `step` in [lo, hi], even over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def _layer(rng):
    """n and k of a layer.  Most model dimensions are multiples of 256; splits of them are sometimes only of 128."""
    n = _log(rng, 512, 57344, 256)
    k = _log(rng, 512, 28672, 256)
    if rng.random() < 0.25:
        k += 128
    return n, k


def draw(rng):
    most = work(listed()[10])
    while True:
        kind = rng.choice(["gemm"] * 6 + ["step", "graph", "host", "pack"])
        case = {"kind": kind, "group": 128 if rng.random() < 0.75 else -1}
        if kind in ("gemm", "pack"):
            case["n"], case["k"] = _layer(rng)
        else:
            case["hidden"] = _log(rng, 1024, 8192, 256)
            case["ffn"] = int(case["hidden"] * rng.uniform(2.2, 3.8)) // 256 * 256
        if kind == "gemm":
            case["m"] = _log(rng, 1, 4096, 1)
            case["call"] = rng.choice(["layer", "mul"])
        elif kind == "step":
            case["m"] = _log(rng, 1, 4096, 1)
        elif kind == "graph":
            case["m"] = _log(rng, 1, 64, 1)
            case["blocks"] = rng.randint(1, 4)
        elif kind == "host":
            case["m"] = _log(rng, 1, 128, 1)
        w = work(case)
        if all(w[x] <= most[x] for x in w):
            return case


def _shapes(case):
    """(n, k) of every layer that one pass goes through."""
    if "n" in case:
        return [(case["n"], case["k"])]
    h, f = case["hidden"], case["ffn"]
    return [(3 * h, h), (h, h), (2 * f, h), (h, f)] * case.get("blocks", 1)


class _Operands:
    """One layer's operands: random codes (every packed word is a valid one), scales and activations of the sizes met
    in quantised models, and the output and lock array that a caller keeps."""

    def __init__(self, gen, m, n, k, group):
        groups = 1 if group == -1 else k // group
        self.A = torch.randn(m, k, generator=gen, device="cuda", dtype=torch.half)
        self.B = torch.randint(-2 ** 31, 2 ** 31, (k // 16, 2 * n), generator=gen, device="cuda", dtype=torch.int)
        self.s = torch.rand(groups, n, generator=gen, device="cuda").mul_(0.015).add_(0.005).half()
        self.C = torch.zeros(m, n, device="cuda", dtype=torch.half)
        self.ws = torch.zeros(n // 128 * 16, device="cuda", dtype=torch.int)

    def mul(self):
        w4.mul(self.A, self.B, self.C, self.s, self.ws)
        return self.C


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind, group = case["kind"], case["group"]
    if kind == "pack":
        n, k = case["n"], case["k"]
        groups = 1 if group == -1 else k // group
        s = torch.rand(groups, n, generator=gen, device="cuda").mul_(0.015).add_(0.005).half()
        w = torch.randint(-8, 8, (n, groups, k // groups), generator=gen, device="cuda", dtype=torch.half)
        w.mul_(s.t().unsqueeze(2))
        return {"kind": kind, "w": w.view(n, k), "s": s, "group": group}
    ops = [_Operands(gen, case["m"], n, k, group) for n, k in _shapes(case)]
    state = {"kind": kind, "ops": ops}
    if kind == "gemm" and case["call"] == "layer":
        state["kind"] = "layer"
        with torch.device("cuda"):
            layer = w4.Layer(case["k"], case["n"], group)
        layer.B.copy_(ops[0].B)
        layer.s.copy_(ops[0].s)
        state["layer"], state["A"] = layer, ops[0].A
        del state["ops"]
    elif kind == "graph":
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):      # the first call on a stream sets its scratch up, which a capture cannot
            for o in ops:
                o.mul()
        torch.cuda.current_stream().wait_stream(stream)
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"], stream=stream):
            for o in ops:
                o.mul()
    elif kind == "host":
        state["host"], state["C"] = [], []
        for o in ops:
            a = o.A.cpu().pin_memory()
            c = torch.zeros(o.C.shape, dtype=torch.half, pin_memory=True)
            state["host"].append(w4.HostGemm(a, o.B, c, o.s, o.ws, o.A, o.C))
            state["C"].append(c)
    return state


def run(state):
    kind = state["kind"]
    if kind == "layer":
        return state["layer"](state["A"])
    if kind == "pack":
        return w4.quantize_pack_device(state["w"], state["s"], state["group"])
    if kind == "graph":
        state["graph"].replay()
        return [o.C for o in state["ops"]]
    if kind == "host":
        for gemm in state["host"]:
            gemm()
        return state["C"]
    return [o.mul() for o in state["ops"]]


def work(case):
    size = flops = 0
    for n, k in _shapes(case):
        groups = 1 if case["group"] == -1 else k // case["group"]
        if case["kind"] == "pack":      # fp16 weights and scales in, packed words and permuted scales out
            size += 2 * n * k + n * k // 2 + 4 * groups * n
        else:                           # packed weights, scales and activations in, outputs out
            size += n * k // 2 + 2 * groups * n + 2 * case["m"] * (n + k)
            flops += 2 * case["m"] * n * k
    return {"bytes": size, "flops": flops}


def tolerance(case):
    """fp16 operands and results, fp32 sums.  Rounding a weight's product with its scale to fp16 or not, and rounding
    the result, are each off by up to 2^-11 of the value, about 2.8e-4 in the mean square; the largest of a hundred
    million such differences lies six or seven standard deviations out, on top of one fp16 step of the result."""
    if case["kind"] == "pack":
        return "exact"
    return {"rel": 1e-3, "max": 6e-3}
