"""The work a program has this package do, as cases that can be timed.

A program that serves a model from GGUF weights calls the package in four ways, and every case is one of them:

* ``linear``: `kernels.gemm_rcr`, one quantized linear or a stack of equal ones (one per layer), with or without bias;
* ``layers``: the quantized linears of decoder layers, called one by one between the attention and norm kernels of the program
  (`kernels.gemm_rcr` for q / k / v / o and down, `kernels.dual_gemm_rcr` for the gated pair); ``mlp``: the gated pair and down alone;
* ``session``: the same layer as a compiled artifact, run with device tensors (`Session.run_torch`, graph replay on, as a decode
  loop with its own buffers does) or with host arrays (``host``: `Session.run_numpy`);
* ``dequantize``: `kernels.dequantize_rows`, a weight expanded to a dense matrix.

M is the number of tokens in flight: 1 for one stream, up to a few dozen for batched decode, hundreds to thousands for prefill.
Weights and activations follow `synthetic.py`; the inputs of gated layers are scaled by K^-1/2 so that the gate sees values of
order one, as it does behind a norm (and so that float16 results stay finite)."""
from __future__ import annotations

import math
import tempfile

import torch

import dinoml_v2_b200 as dml
from dinoml_v2_b200 import kernels, synthetic
from dinoml_v2_b200.constant_sources import GGUFConstant
from dinoml_v2_b200.gguf_blocks import encoded_nbytes, qtype_of

ELEMENT_BYTES = {"float16": 2, "bfloat16": 2, "float32": 4}
MAX_M = 2048
MAX_HIDDEN, MAX_FFN = 8192, 28672


def listed():
    return [
        # the smallest call: one Q8_0 projection, float32 activations, one token - the latency of a single call
        {"name": "one_call_q8_0_f32", "kind": "linear", "qtype": "Q8_0", "dtype": "float32", "m": 1, "n": 4096, "k": 4096, "count": 1, "bias": False},
        # decode, one stream: the same up-projection in six layers (every pass reads more weights than the L2 holds)
        {"name": "decode_q4_k", "kind": "linear", "qtype": "Q4_K", "dtype": "bfloat16", "m": 1, "n": 11008, "k": 4096, "count": 6, "bias": False},
        # decode, one stream: all quantized linears of four decoder layers with the usual Q4_K / Q6_K mix
        {"name": "decode_layers", "kind": "layers", "qtype": "Q4_K", "qtype_down": "Q6_K", "dtype": "bfloat16", "m": 1, "hidden": 4096, "kv": 1024,
         "ffn": 14336, "count": 4},
        # the same layer as a compiled artifact on device tensors
        {"name": "decode_session", "kind": "session", "qtype": "Q4_K", "qtype_down": "Q6_K", "dtype": "bfloat16", "m": 1, "hidden": 4096, "kv": 1024,
         "ffn": 14336, "count": 1, "host": False},
        # a small batch served through host arrays; the down projection's rows (K = 11008) are not multiples of 16 bytes
        {"name": "host_session_m4", "kind": "session", "qtype": "Q4_K", "qtype_down": "Q6_K", "dtype": "float16", "m": 4, "hidden": 4096, "kv": 4096,
         "ffn": 11008, "count": 1, "host": True},
        # batched decode on the largest MLP
        {"name": "batch_mlp_m16", "kind": "mlp", "qtype": "Q4_K", "qtype_down": "Q4_K", "dtype": "bfloat16", "m": 16, "hidden": 8192, "ffn": 28672, "count": 1},
        # batched decode on 32-weight blocks: K is no multiple of 256, with bias, in four layers
        {"name": "batch_mxfp4_bias_m24", "kind": "linear", "qtype": "MXFP4", "dtype": "bfloat16", "m": 24, "n": 5760, "k": 2880, "count": 4, "bias": True},
        # a short prompt through one decoder layer
        {"name": "chunk_layer_m100", "kind": "layers", "qtype": "Q4_K", "qtype_down": "Q6_K", "dtype": "bfloat16", "m": 100, "hidden": 4096, "kv": 1024,
         "ffn": 14336, "count": 1},
        # prefill of 512 tokens, one down projection
        {"name": "prefill_q6_k_m512", "kind": "linear", "qtype": "Q6_K", "dtype": "bfloat16", "m": 512, "n": 4096, "k": 14336, "count": 1, "bias": False},
        # prefill of an odd number of tokens, the MLP with K = 11008 in its down projection
        {"name": "prefill_mlp_m333", "kind": "mlp", "qtype": "Q4_K", "qtype_down": "Q6_K", "dtype": "float16", "m": 333, "hidden": 4096, "ffn": 11008, "count": 1},
        # the largest: a long prefill through the largest MLP
        {"name": "prefill_mlp_m2048", "kind": "mlp", "qtype": "Q4_K", "qtype_down": "Q6_K", "dtype": "bfloat16", "m": 2048, "hidden": 8192, "ffn": 28672,
         "count": 1},
        # a weight expanded to dense float16
        {"name": "dequantize_q4_k_f16", "kind": "dequantize", "qtype": "Q4_K", "dtype": "float16", "n": 11008, "k": 4096},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _multiple(rng, low, high, step):
    return max(1, int(round(_log_int(rng, low, high) / step))) * step


def draw(rng):
    """One more case of the same ranges: every weight type (the three common ones more often), every activation type, M and the
    matrix sizes spread over their logarithms, N of any residue, K at the multiples the weight type allows."""
    kind = rng.choices(["linear", "mlp", "layers", "session", "dequantize"], [40, 20, 12, 16, 12])[0]
    qtype = rng.choices(["Q4_K", "Q6_K", "Q8_0", "Q5_K", "Q4_0", "Q3_K", "Q2_K", "MXFP4", "NVFP4"], [8, 5, 5, 2, 2, 2, 2, 2, 2])[0]
    dtype = rng.choices(["bfloat16", "float16", "float32"], [6, 3, 1])[0]
    if kind in ("linear", "dequantize"):
        block = qtype_of(qtype).block_size
        # models with 32-weight blocks are the ones whose K is not a multiple of 256; most still are
        step = 256 if block == 256 or rng.random() < 0.7 else block
        n, k = _log_int(rng, 256, 32768), _multiple(rng, 1024, 16384, step)
        if kind == "dequantize":
            return {"kind": kind, "qtype": qtype, "dtype": dtype, "n": n, "k": k}
        m = _log_int(rng, 1, MAX_M)
        # shapes without 16-byte weight rows and float32 activations come in smaller sizes, as they do in use
        cap = 1 << (31 if dtype == "float32" or (k // block * qtype_of(qtype).block_bytes) % 16 else 38)
        while m > 1 and m * n * k > cap:
            m = (m + 1) // 2
        count = rng.randint(1, 6) if m <= 16 else 1
        return {"kind": kind, "qtype": qtype, "dtype": dtype, "m": m, "n": n, "k": k, "count": count, "bias": rng.random() < 0.3}
    # gated layers: 16-bit activations, 256-weight multiples
    dtype = dtype if dtype != "float32" else "bfloat16"
    hidden, ffn = _multiple(rng, 1024, MAX_HIDDEN, 256), _multiple(rng, 2816, MAX_FFN, 256)
    if qtype in ("Q2_K", "Q3_K", "MXFP4"):          # the gated kernels take these where weight rows are multiples of 16 bytes
        hidden = max(2048, hidden // 2048 * 2048)
    if qtype == "Q6_K":
        hidden = max(2048, hidden // 2048 * 2048)
    down = "Q6_K" if rng.random() < 0.5 else "Q4_K"
    case = {"kind": kind, "qtype": qtype, "qtype_down": down, "dtype": dtype, "hidden": hidden, "ffn": ffn, "count": 1}
    if kind == "session":
        hidden, ffn = min(hidden, 4096), min(ffn, 14336)     # an artifact carries its weights through the host: one moderate layer
        case.update(hidden=hidden, ffn=ffn, kv=max(256, hidden // rng.choice([1, 4, 8]) // 256 * 256), m=_log_int(rng, 1, 128), host=rng.random() < 0.4)
    else:
        case.update(m=_log_int(rng, 1, MAX_M))
        if kind == "layers":
            case.update(kv=max(256, hidden // rng.choice([1, 4, 8]) // 256 * 256))
        # down projections without 16-byte weight rows (Q6_K, K not a multiple of 2048)
        while down == "Q6_K" and ffn % 2048 and case["m"] > 16 and case["m"] * hidden * ffn > 1 << 34:
            case["m"] = (case["m"] + 1) // 2
        if case["m"] <= 16:
            case["count"] = rng.randint(1, 3)
    return case


# ----------------------------------------------------------------------------------------------- sizes
def _matrices(case):
    """(qtype, rows, K, output columns) of every quantized linear of one pass."""
    if case["kind"] in ("linear", "dequantize"):
        return [(case["qtype"], case["n"], case["k"], case["n"])] * case.get("count", 1)
    h, f, q, down = case["hidden"], case["ffn"], case["qtype"], case["qtype_down"]
    one = [] if case["kind"] == "mlp" else [(q, h, h, h), (q, case["kv"], h, case["kv"]), (q, case["kv"], h, case["kv"]), (q, h, h, h)]
    return (one + [(q, 2 * f, h, f), (down, h, f, h)]) * case["count"]


def work(case):
    e = ELEMENT_BYTES[case["dtype"]]
    weights = sum(encoded_nbytes(q, n, k) for q, n, k, _ in _matrices(case))
    if case["kind"] == "dequantize":
        return {"bytes": weights + case["n"] * case["k"] * e, "flops": case["n"] * case["k"]}
    m = case["m"]
    flops = sum(2 * m * n * k for _, n, k, _ in _matrices(case))
    if case["kind"] == "linear":
        dense = case["count"] * (m * case["k"] + m * case["n"] + (case["n"] if case["bias"] else 0))
    elif case["kind"] == "mlp":                                  # x in, result out; the gated activations stay inside
        dense = case["count"] * 2 * m * case["hidden"]
    else:                                                        # x, attention output, MLP input; q, k, v, o and the MLP's result
        dense = case["count"] * m * (6 * case["hidden"] + 2 * case["kv"])
    if case.get("host"):                                         # host arrays: every value also crosses the bus
        dense *= 2
    return {"bytes": weights + e * dense, "flops": flops}


def tolerance(case):
    if case["kind"] == "dequantize":
        return "exact"
    return {"rel": {"float32": 1e-5, "float16": 2e-3, "bfloat16": 1e-2}[case["dtype"]]}


# ----------------------------------------------------------------------------------------------- inputs
class _Maker:
    def __init__(self, case, seed):
        self.dev, self.seed, self.dtype = torch.device("cuda"), int(seed) * 1000, getattr(torch, case["dtype"])
        self.generator = torch.Generator(device=self.dev)
        self.generator.manual_seed(self.seed)

    def blocks(self, qtype, n, k):
        self.seed += 1
        return synthetic.random_blocks_torch(qtype, n, k, self.seed, self.dev)

    def dense(self, *shape, scale=1.0):
        return (torch.randn(*shape, device=self.dev, generator=self.generator) * scale).to(self.dtype)


def _layer_inputs(make, case):
    scale = case["hidden"] ** -0.5
    return {name: make.dense(case["m"], case["hidden"], scale=scale) for name in ("x", "attn", "x2")}


class _Layer(dml.Module):
    """The quantized linears of one decoder layer, as a program writes them for `dml.compile`."""

    def __init__(self, case):
        h, kv, f, dt = case["hidden"], case["kv"], case["ffn"], case["dtype"]
        self.q, self.k, self.v, self.o = (dml.Parameter([n, h], dtype=dt) for n in (h, kv, kv, h))
        self.gate, self.up, self.down = dml.Parameter([f, h], dtype=dt), dml.Parameter([f, h], dtype=dt), dml.Parameter([h, f], dtype=dt)

    def forward(self, x, attn, x2):
        ops = dml.ops
        return [ops.gemm_rcr(x, self.q), ops.gemm_rcr(x, self.k), ops.gemm_rcr(x, self.v), ops.gemm_rcr(attn, self.o),
                ops.gemm_rcr(ops.dual_gemm_rcr_silu(x2, self.gate, self.up), self.down)]


def _prepare_session(make, case):
    h, kv, f = case["hidden"], case["kv"], case["ffn"]
    shapes = {"q": (h, h), "k": (kv, h), "v": (kv, h), "o": (h, h), "gate": (f, h), "up": (f, h), "down": (h, f)}
    constants = {}
    for name, (n, k) in shapes.items():
        qtype = case["qtype_down"] if name == "down" else case["qtype"]
        constants[name] = GGUFConstant.from_blocks(make.blocks(qtype, n, k).cpu().numpy(), qtype, (n, k), tensor=name)
    tokens = dml.Dim("tokens", 1, max(128, case["m"]))
    spec = dml.trace(_Layer(case), inputs={name: dml.TensorSpec([tokens, h], case["dtype"]) for name in ("x", "attn", "x2")}, constants=constants)
    folder = tempfile.TemporaryDirectory(prefix="artifact_")
    module = dml.runtime.load(dml.compile(spec, dml.Target("cuda"), folder.name).path)
    module.load_encoded_constants()
    session = module.create_session()
    state = {"kind": "host" if case["host"] else "session", "session": session, "module": module, "folder": folder}
    inputs = _layer_inputs(make, case)
    if case["host"]:
        # bfloat16 travels as float32 arrays, as numpy has no such type
        state["inputs"] = {name: (t.float() if case["dtype"] == "bfloat16" else t).cpu().numpy() for name, t in inputs.items()}
        return state
    names = [o["name"] for o in module.metadata["outputs"]]
    state["inputs"] = inputs
    state["outputs"] = {name: torch.empty(case["m"], n, dtype=make.dtype, device=make.dev) for name, n in zip(names, (h, kv, kv, h, h))}
    session.set_graph_replay(True)
    return state


def prepare(case, seed):
    make = _Maker(case, seed)
    kind = case["kind"]
    if kind == "session":
        return _prepare_session(make, case)
    if kind == "dequantize":
        return {"kind": kind, "qtype": case["qtype"], "dtype": case["dtype"], "k": case["k"], "w": make.blocks(case["qtype"], case["n"], case["k"])}
    if kind == "linear":
        n, k = case["n"], case["k"]
        return {"kind": kind, "qtype": case["qtype"],
                "layers": [(make.dense(case["m"], k), make.blocks(case["qtype"], n, k), make.dense(n) if case["bias"] else None) for _ in range(case["count"])]}
    h, f, q, down = case["hidden"], case["ffn"], case["qtype"], case["qtype_down"]
    layers = []
    for _ in range(case["count"]):
        layer = {"in": _layer_inputs(make, case), "gate_up": kernels.interleave_rows8(make.blocks(q, f, h), make.blocks(q, f, h)), "down": make.blocks(down, h, f)}
        if kind == "layers":
            layer.update(q=make.blocks(q, h, h), k=make.blocks(q, case["kv"], h), v=make.blocks(q, case["kv"], h), o=make.blocks(q, h, h))
        layers.append(layer)
    return {"kind": kind, "qtype": q, "qtype_down": down, "layers": layers}


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return [kernels.gemm_rcr(x, w, state["qtype"], bias) for x, w, bias in state["layers"]]
    if kind == "dequantize":
        return kernels.dequantize_rows(state["w"], state["qtype"], state["k"], state["dtype"])
    if kind == "session":
        return state["session"].run_torch(state["inputs"], state["outputs"])
    if kind == "host":
        return state["session"].run_numpy(state["inputs"])
    q, out = state["qtype"], []
    for layer in state["layers"]:
        inputs = layer["in"]
        if kind == "layers":
            out += [kernels.gemm_rcr(inputs["x"], layer["q"], q), kernels.gemm_rcr(inputs["x"], layer["k"], q), kernels.gemm_rcr(inputs["x"], layer["v"], q),
                    kernels.gemm_rcr(inputs["attn"], layer["o"], q)]
        out.append(kernels.gemm_rcr(kernels.dual_gemm_rcr(inputs["x2"], layer["gate_up"], q, "silu"), layer["down"], state["qtype_down"]))
    return out
