"""Performance cases of the packed-ternary matmul path: what is timed, on which inputs, and how exact it has to be.

Every case is work that a user of the package asks for through its public entry points:

  linear    one eval-mode ternary ``Linear`` forward of a converted model, from one token (decode, latency) to a long
            prompt (prefill, tensor cores)
  decode    one decode step through the Linears of decoder blocks, each reading the one before; replayed from a CUDA
            graph, as a serving loop does, or called eagerly
  quantize  ``TernaryTensor.from_float``: threshold-quantise and pack a weight matrix
  train     one quantisation-aware training step of a ``Linear``: forward, and the gradients of input, weight and bias
  tq        GGUF ternary blocks: export of packed weights and import of the blocks again
  gemm      ``t81lib.gemm_ternary`` (C = alpha A B + beta C) with dense B, on host buffers or on the device

``listed()`` names the sizes followed over time, ``draw()`` gives others of the same ranges.  Layer shapes are those of
the benchmark: Llama-3-8B-shaped (hidden 4096, FFN 14336, 1024 key/value features) and Phi-3-mini-shaped (hidden 3072,
FFN 8192, fused qkv and gate/up).  Weights are N(0, 0.02^2) under the absmean rule, activations N(0, 1).
Packed operands on both sides of ``gemm_ternary`` (whole-limb integer products) overflow fp32 beyond toy sizes and are
not a workload.
"""

import math

import torch
from torch import nn

from t81lib_b200 import ops, t81lib
from t81lib_b200 import torch as t81_torch
from t81lib_b200.convert import convert_module
from t81lib_b200.nn import Linear

_DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16, "float16": torch.float16}
_SIZE = {"float32": 4, "bfloat16": 2, "float16": 2}
_THRESHOLD = 0.45

# what the largest listed cases cost; drawn ones stay below
_MOST_LINEAR = 2.0 * 16384 * 4096 * 14336
_MOST_TRAIN = 2.0 * 4096 * 4096 * 14336
_MOST_WEIGHTS = 14336 * 4096


def listed():
    return [
        # the smallest call: one token through an attention output projection, where launch and host latency count
        {"name": "linear_3072x3072_1tok", "kind": "linear", "tokens": 1, "in": 3072, "out": 3072, "dtype": "bfloat16",
         "bias": False},
        # a serving step at batch 8: two decoder blocks (14 Linears) from a CUDA graph, weights streamed from HBM
        {"name": "decode_2x4096_8tok_graph", "kind": "decode", "tokens": 8, "hidden": 4096, "kv": 1024, "ffn": 14336,
         "blocks": 2, "fused": False, "dtype": "bfloat16", "graph": True},
        # the same without a graph, an odd batch and fp16: fused qkv and gate/up, whose consumers read column slices
        {"name": "decode_1x3072_13tok_fp16", "kind": "decode", "tokens": 13, "hidden": 3072, "kv": 3072, "ffn": 8192,
         "blocks": 1, "fused": True, "dtype": "float16", "graph": False},
        # between decode and prefill: a large batch, a short prompt or a speculated continuation
        {"name": "linear_14336x4096_80tok", "kind": "linear", "tokens": 80, "in": 4096, "out": 14336,
         "dtype": "bfloat16", "bias": False},
        # an ordinary prompt with bias
        {"name": "linear_9216x3072_2048tok", "kind": "linear", "tokens": 2048, "in": 3072, "out": 9216,
         "dtype": "bfloat16", "bias": True},
        # the largest: eight 2048-token prompts at once through the long contraction
        {"name": "linear_4096x14336_16384tok", "kind": "linear", "tokens": 16384, "in": 14336, "out": 4096,
         "dtype": "bfloat16", "bias": False},
        # fp32 activations (a model that was not cast down), nothing a multiple of anything
        {"name": "linear_1999x3001_777tok_fp32", "kind": "linear", "tokens": 777, "in": 3001, "out": 1999,
         "dtype": "float32", "bias": True},
        # converting a checkpoint: one weight matrix
        {"name": "quantize_4096x4096_absmean", "kind": "quantize", "rows": 4096, "cols": 4096, "dtype": "float32",
         "rule": "absmean"},
        # quantisation-aware training with bf16 activations over fp32 master weights
        {"name": "train_14336x4096_4096tok_bf16", "kind": "train", "tokens": 4096, "in": 4096, "out": 14336,
         "dtype": "bfloat16", "bias": False},
        # the same in fp32 throughout (the layer's default), a small ragged layer
        {"name": "train_2050x1537_1000tok_fp32", "kind": "train", "tokens": 1000, "in": 1537, "out": 2050,
         "dtype": "float32", "bias": True},
        # a GGUF export of a packed layer and the import of the file's blocks
        {"name": "tq1_14336x4096", "kind": "tq", "rows": 14336, "cols": 4096, "format": "TQ1_0"},
        # the drop-in module call on numpy buffers, updating C in place
        {"name": "gemm_512x256x528_host", "kind": "gemm", "M": 512, "N": 256, "K": 528, "beta": 0.5, "host": True},
    ]


def _between(rng, lo, hi):
    """A size spread over the logarithm of [lo, hi]: as it comes (odd ones among them) or, as often, a round one."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    step = rng.choice((1, 1, 16, 128))
    return max(lo, min(hi, (n + step - 1) // step * step))


def draw(rng):
    kind = rng.choice(("linear", "linear", "linear", "linear", "decode", "decode", "quantize", "train", "train", "tq", "gemm"))
    dtype = rng.choice(("bfloat16", "bfloat16", "float16", "float32"))
    if kind == "linear":
        fan_in, fan_out, tokens = _between(rng, 512, 14336), _between(rng, 512, 14336), _between(rng, 1, 16384)
        tokens = max(1, min(tokens, int(_MOST_LINEAR / (2.0 * fan_in * fan_out) / (1 if _SIZE[dtype] == 2 else 2))))
        return {"kind": kind, "tokens": tokens, "in": fan_in, "out": fan_out, "dtype": dtype, "bias": rng.random() < 0.5}
    if kind == "decode":
        hidden, ffn, fused = _between(rng, 1024, 4096), _between(rng, 2048, 14336), rng.random() < 0.5
        return {"kind": kind, "tokens": rng.randint(1, 16), "hidden": hidden, "kv": hidden if rng.random() < 0.5 else max(256, hidden // 4),
                "ffn": ffn, "blocks": rng.randint(1, 2), "fused": fused, "dtype": dtype, "graph": rng.random() < 0.5}
    if kind == "quantize":
        rows, cols = _between(rng, 512, 14336), _between(rng, 512, 14336)
        return {"kind": kind, "rows": max(1, min(rows, _MOST_WEIGHTS // cols)), "cols": cols, "dtype": dtype,
                "rule": rng.choice(("absmean", "absmean", "fixed"))}
    if kind == "train":
        fan_in, fan_out, tokens = _between(rng, 512, 14336), _between(rng, 512, 14336), _between(rng, 256, 8192)
        tokens = max(1, min(tokens, int(_MOST_TRAIN / (2.0 * fan_in * fan_out))))
        return {"kind": kind, "tokens": tokens, "in": fan_in, "out": fan_out, "dtype": "bfloat16" if dtype == "float16" else dtype,
                "bias": rng.random() < 0.5}
    if kind == "tq":
        rows, cols = _between(rng, 512, 14336), _between(rng, 512, 14336)
        return {"kind": kind, "rows": max(1, min(rows, _MOST_WEIGHTS // cols)), "cols": cols, "format": rng.choice(("TQ1_0", "TQ2_0"))}
    return {"kind": "gemm", "M": _between(rng, 128, 2048), "N": _between(rng, 128, 2048), "K": 48 * rng.randint(4, 64),
            "beta": rng.choice((0.0, 0.5)), "host": rng.random() < 0.5}


def _normal(gen, *shape, std=1.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float32) * std).to(dtype)


def _float_linear(gen, fan_in, fan_out, bias):
    layer = nn.utils.skip_init(nn.Linear, fan_in, fan_out, bias=bias, device="cuda")
    with torch.no_grad():
        layer.weight.copy_(_normal(gen, fan_out, fan_in, std=0.02))
        if bias:
            layer.bias.copy_(_normal(gen, fan_out, std=0.01))
    return layer


def _deploy(model):
    """An inference deployment: packed weights only, nothing that records gradients."""
    convert_module(model, threshold=_THRESHOLD, rule="absmean", release_float=True, verbose=False)
    return model.eval().requires_grad_(False)


class _Block(nn.Module):
    """The Linears of a decoder block in their order of use; what lies between them is not part of this package."""

    def __init__(self, gen, hidden, kv, ffn, fused):
        super().__init__()
        self.hidden, self.ffn, self.fused = hidden, ffn, fused
        if fused:
            self.qkv = _float_linear(gen, hidden, hidden + 2 * kv, False)
            self.gate_up = _float_linear(gen, hidden, 2 * ffn, False)
        else:
            self.q = _float_linear(gen, hidden, hidden, False)
            self.k = _float_linear(gen, hidden, kv, False)
            self.v = _float_linear(gen, hidden, kv, False)
            self.gate = _float_linear(gen, hidden, ffn, False)
            self.up = _float_linear(gen, hidden, ffn, False)
        self.o = _float_linear(gen, hidden, hidden, False)
        self.down = _float_linear(gen, ffn, hidden, False)

    def forward(self, x):
        if self.fused:
            qkv = self.qkv(x)
            gate_up = self.gate_up(self.o(qkv[:, :self.hidden]))
            return self.down(gate_up[:, :self.ffn]), (qkv, gate_up)
        q, k, v = self.q(x), self.k(x), self.v(x)
        attended = self.o(q)
        gate, up = self.gate(attended), self.up(attended)
        return self.down(gate), (k, v, up)


def _decode_step(blocks, x, scale):
    outputs = []
    for block in blocks:
        y, rest = block(x)
        outputs.extend((y, *rest))
        x = y * scale  # stands for the normalisation between blocks, and keeps fp16 in range
    return outputs


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "linear":
        model = nn.Sequential(_float_linear(gen, case["in"], case["out"], case["bias"]))
        x = _normal(gen, case["tokens"], case["in"], dtype=_DTYPES[case["dtype"]])
        return {"kind": kind, "layer": _deploy(model)[0], "x": x}
    if kind == "decode":
        model = _deploy(nn.ModuleList(_Block(gen, case["hidden"], case["kv"], case["ffn"], case["fused"])
                                      for _ in range(case["blocks"])))
        x = _normal(gen, case["tokens"], case["hidden"], std=0.25, dtype=_DTYPES[case["dtype"]])
        state = {"kind": kind, "blocks": model, "x": x, "scale": 1.0 / 32.0, "graph": None}
        if case["graph"]:
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                _decode_step(model, x, state["scale"])
            torch.cuda.current_stream().wait_stream(side)
            state["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(state["graph"]):
                state["outputs"] = _decode_step(model, x, state["scale"])
        return state
    if kind == "quantize":
        # the fixed threshold compares the weights themselves, so they come normalised
        std = 0.02 if case["rule"] == "absmean" else 0.5
        w = _normal(gen, case["rows"], case["cols"], std=std, dtype=_DTYPES[case["dtype"]])
        return {"kind": kind, "w": w, "rule": case["rule"]}
    if kind == "train":
        layer = Linear(case["in"], case["out"], bias=case["bias"], device="cuda", threshold=_THRESHOLD)
        with torch.no_grad():
            layer.weight.copy_(_normal(gen, case["out"], case["in"], std=0.02))
            if case["bias"]:
                layer.bias.copy_(_normal(gen, case["out"], std=0.01))
        dtype = _DTYPES[case["dtype"]]
        x = _normal(gen, case["tokens"], case["in"], dtype=dtype).requires_grad_(True)
        grad = _normal(gen, case["tokens"], case["out"], std=0.05, dtype=dtype)
        return {"kind": kind, "layer": layer.train(), "x": x, "grad": grad}
    if kind == "tq":
        w = _normal(gen, case["rows"], case["cols"], std=0.02)
        t = t81_torch.TernaryTensor.from_float(w, threshold=_THRESHOLD, rule="absmean")
        return {"kind": kind, "packed": t.packed, "scale": t.row_scale, "rows": case["rows"], "cols": case["cols"], "format": case["format"]}
    M, N, K = case["M"], case["N"], case["K"]
    a = t81lib.pack_dense_matrix(_normal(gen, M, K, std=0.5), _THRESHOLD)
    b, c = _normal(gen, K, N), _normal(gen, M, N)
    if case["host"]:
        a, b, c = a.cpu().numpy(), b.cpu().numpy(), c.cpu().numpy()
    return {"kind": "gemm", "a": a, "b": b, "c": c, "M": M, "N": N, "K": K, "beta": case["beta"]}


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["layer"](state["x"])
    if kind == "decode":
        if state["graph"] is not None:
            state["graph"].replay()
            return state["outputs"]
        return _decode_step(state["blocks"], state["x"], state["scale"])
    if kind == "quantize":
        t = t81_torch.TernaryTensor.from_float(state["w"], threshold=_THRESHOLD, rule=state["rule"])
        return [t.packed, t.row_scale]
    if kind == "train":
        layer, x = state["layer"], state["x"]
        y = layer(x)
        wanted = [x, layer.weight] + ([layer.bias] if layer.bias is not None else [])
        return [y.detach(), *torch.autograd.grad(y, wanted, state["grad"]), layer.training_scale]
    if kind == "tq":
        blocks = ops.packed_to_tq(state["packed"], state["rows"], state["cols"], state["format"], state["scale"])
        return [blocks, *ops.tq_to_packed(blocks, state["rows"], state["cols"], state["format"])]
    t81lib.gemm_ternary(state["a"], state["b"], state["c"], state["M"], state["N"], state["K"], 1.0, state["beta"])
    return state["c"]


def _linear_work(tokens, fan_in, fan_out, size):
    """Two bits a weight, its row scale, activations in, results out."""
    return (fan_in * fan_out / 4.0 + 4.0 * fan_out + size * tokens * (fan_in + fan_out), 2.0 * tokens * fan_in * fan_out)


def work(case):
    kind = case["kind"]
    if kind == "linear":
        nbytes, flops = _linear_work(case["tokens"], case["in"], case["out"], _SIZE[case["dtype"]])
        return {"bytes": nbytes + (4.0 * case["out"] if case["bias"] else 0.0), "flops": flops}
    if kind == "decode":
        h, kv, f = case["hidden"], case["kv"], case["ffn"]
        layers = [(h, h + 2 * kv), (h, h), (h, 2 * f), (f, h)] if case["fused"] else \
            [(h, h), (h, kv), (h, kv), (h, h), (h, f), (h, f), (f, h)]
        each = [_linear_work(case["tokens"], i, o, _SIZE[case["dtype"]]) for i, o in layers]
        return {"bytes": case["blocks"] * sum(b for b, _ in each), "flops": case["blocks"] * sum(n for _, n in each)}
    if kind == "quantize":
        rows, cols = case["rows"], case["cols"]
        return {"bytes": float(rows) * (cols * _SIZE[case["dtype"]] + 16 * ((cols + 47) // 48) + (4 if case["rule"] == "absmean" else 0)), "flops": 0.0}
    if kind == "train":
        t, i, o, size = case["tokens"], case["in"], case["out"], _SIZE[case["dtype"]]
        # x and the output's gradient in, y and x's gradient out, the weight in and its gradient out
        return {"bytes": 2.0 * size * t * (i + o) + 8.0 * i * o, "flops": 3 * 2.0 * t * i * o}
    if kind == "tq":
        rows, cols = case["rows"], case["cols"]
        blocks = (cols + 255) // 256
        packed, payload = rows * 16.0 * ((cols + 47) // 48), rows * blocks * (54.0 if case["format"] == "TQ1_0" else 66.0)
        return {"bytes": 2 * packed + 2 * payload + 4.0 * rows * (1 + blocks), "flops": 0.0}
    M, N, K = case["M"], case["N"], case["K"]
    return {"bytes": M * K / 3.0 + 4.0 * K * N + (8.0 if case["beta"] else 4.0) * M * N, "flops": 2.0 * M * N * K}


def tolerance(case):
    kind = case["kind"]
    if kind in ("quantize", "tq"):
        return "exact"
    # exact products, fp32 accumulation; 16-bit results are rounded once per Linear, and in a chain each rounding is
    # the next one's input.  fp32 activations enter the products with at least 16 mantissa bits.
    rel = {"bfloat16": 1e-2, "float16": 1.5e-3, "float32": 3e-5}[case.get("dtype", "float32")]
    return {"rel": rel}
