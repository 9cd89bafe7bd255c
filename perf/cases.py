"""The measured workloads: what users of this package have it do, through its public entry points.

Five kinds of work, each over the sizes it meets in use:
  linear      one QuantizedLinear.forward: a projection called eagerly, batch 1 to 2048
  blocks      gated MLP blocks (gate/up with SiLU, then down), one after the other, as a decoder's layers run them;
              small batches as one captured CUDA graph (a decoding loop), larger ones as eager calls (prefill)
  stack       several Linears with f32 activations in one pass: a chained classifier, or the projections of a GPT
  quantize    quantize_tensor of one weight, or quantize_named_parameters of a model
  dequantize  dequantize_tensor of one weight
"""
import math

import torch

from shrew_b200 import (Linear, QuantBits, QuantConfig, QuantGranularity, QuantizedLinear, QuantMode, dequantize_tensor,
                        quantize_named_parameters, quantize_tensor)
from shrew_b200 import _lib

_DTYPE = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
_SIZE = {"f32": 4, "bf16": 2, "f16": 2}


def listed():
    return [
        # the smallest call: a 784 -> 256 -> 10 classifier on a batch of 64, all launch latency and host path
        dict(name="mlp_784_256_10_b64", kind="stack", shape="classifier", m=64, d_in=784, d_hidden=256, d_out=10),
        # one projection for one token: a decoding step of an eager program
        dict(name="linear_4096_m1", kind="linear", n=4096, k=4096, m=1, x="bf16", y="bf16", weights="int8",
             granularity="channel", bias=True, relu=False),
        # the same projection for 16 sequences decoded together, weights quantized with one scale
        dict(name="linear_4096_m16", kind="linear", n=4096, k=4096, m=16, x="bf16", y="bf16", weights="int8",
             granularity="tensor", bias=False, relu=False),
        # a short prompt of ragged length through one projection
        dict(name="linear_4096_m250", kind="linear", n=4096, k=4096, m=250, x="bf16", y="bf16", weights="int8",
             granularity="channel", bias=True, relu=False),
        # token-by-token decoding through four Llama-sized MLP blocks: bound by the weight stream
        dict(name="blocks_decode_m1", kind="blocks", layers=4, d=4096, ff=11008, m=1, graph=True),
        # decoding of 24 sequences together through two such blocks
        dict(name="blocks_decode_m24", kind="blocks", layers=2, d=4096, ff=11008, m=24, graph=True),
        # prefill of 512 tokens through one block: bound by the tensor cores
        dict(name="block_prefill_m512", kind="blocks", layers=1, d=4096, ff=11008, m=512, graph=False),
        # the 25 Linears of a small GPT (width 256, 4 blocks, vocabulary 50257) on 8 x 512 tokens of f32 activations
        dict(name="tinygpt_stack_m4096", kind="stack", shape="gpt", m=4096, d=256, ff=1024, blocks=4, vocab=50257),
        # quantization of one large f32 weight, per channel
        dict(name="quantize_f32_8192x8192", kind="quantize", rows=8192, cols=8192, x="f32", bits=8, mode="symmetric",
             granularity="channel"),
        # the same step for a checkpoint that is stored in bf16
        dict(name="quantize_bf16_11008x4096", kind="quantize", rows=11008, cols=4096, x="bf16", bits=8, mode="symmetric",
             granularity="channel"),
        # a whole small model at once: many little matrices
        dict(name="quantize_tinygpt", kind="model", d=256, ff=1024, blocks=4, vocab=50257, granularity="channel"),
        # the way back: an embedding-sized weight to f32
        dict(name="dequantize_50257x256", kind="dequantize", rows=50257, cols=256, y="f32", granularity="channel"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _width(rng, lo, hi):
    """A layer width: mostly a multiple of 64, as model widths are, sometimes only of 16, sometimes any number."""
    v, r = _log_int(rng, lo, hi), rng.random()
    step = 64 if r < 0.7 else (16 if r < 0.85 else 1)
    return max(step, v // step * step)


def draw(rng):
    kind = rng.choices(["linear", "blocks", "classifier", "gpt", "quantize", "model", "dequantize"], [6, 3, 2, 1, 4, 1, 2])[0]
    gran = rng.choice(["channel", "channel", "tensor"])
    if kind == "linear":
        n, k, m = _width(rng, 64, 16384), _width(rng, 64, 11008), _log_int(rng, 1, 2048)
        n = min(n, (1 << 26) // k)
        m = max(1, min(m, (1 << 35) // (n * k) if k % 16 == 0 else (1 << 30) // (n * k)))
        x = rng.choice(["bf16", "bf16", "f32"])
        weights = "int8"
        if x == "bf16" and m <= 32 and k % 128 == 0 and rng.random() < 0.2:
            weights = "int4"
        return dict(kind="linear", n=n, k=k, m=m, x=x, y="f32" if rng.random() < 0.2 else x, weights=weights,
                    granularity=gran, bias=rng.random() < 0.5, relu=rng.random() < 0.25)
    if kind == "blocks":
        m = _log_int(rng, 1, 1024)
        d = _log_int(rng, 512, 5120) // 64 * 64
        ff = int(d * rng.choice([2.6875, 3.5, 4])) // 64 * 64
        layers = rng.randint(1, 4) if m <= 64 else 1
        return dict(kind="blocks", layers=layers, d=d, ff=ff, m=m, graph=m <= 64)
    if kind == "classifier":
        return dict(kind="stack", shape="classifier", m=_log_int(rng, 1, 1024), d_in=_width(rng, 16, 3072),
                    d_hidden=_width(rng, 32, 2048), d_out=_log_int(rng, 2, 1000))
    if kind == "gpt":
        d = rng.randint(2, 8) * 64
        m, vocab = _log_int(rng, 256, 4096), _log_int(rng, 2000, 50257)
        return dict(kind="stack", shape="gpt", m=m, d=d, ff=4 * d, blocks=rng.randint(1, 4), vocab=min(vocab, (1 << 27) // m))
    if kind == "quantize":
        rows, cols = _width(rng, 128, 32768), _width(rng, 128, 16384)
        rows = max(1, min(rows, (1 << 27) // cols))
        return dict(kind="quantize", rows=rows, cols=cols, x=rng.choice(["f32", "f32", "f32", "bf16", "bf16", "f16"]),
                    bits=rng.choice([8, 8, 8, 4]), mode=rng.choice(["symmetric", "symmetric", "symmetric", "asymmetric"]),
                    granularity=gran)
    if kind == "model":
        d = rng.randint(2, 12) * 64
        return dict(kind="model", d=d, ff=4 * d, blocks=rng.randint(1, 4), vocab=_log_int(rng, 1000, 50257), granularity=gran)
    rows, cols = _width(rng, 128, 32768), _width(rng, 128, 16384)
    return dict(kind="dequantize", rows=max(1, min(rows, (1 << 27) // cols)), cols=cols, y=rng.choice(["f32", "f32", "bf16"]),
                granularity=gran)


# ---- the parts of a case ----------------------------------------------------------------------------------------
def _gpt_layers(case):
    """(out, in, relu) of a GPT's Linears: q, k, v, o, up, down per block, then the vocabulary head."""
    d, ff = case["d"], case["ff"]
    return ([(d, d, False)] * 4 + [(ff, d, True), (d, ff, False)]) * case["blocks"] + [(case["vocab"], d, False)]


def _config(case):
    cfg = QuantConfig(QuantBits.Int4 if case.get("bits", 8) == 4 else QuantBits.Int8, QuantMode.Symmetric,
                      QuantGranularity.PerTensor if case["granularity"] == "tensor" else QuantGranularity.PerChannel)
    return cfg.asymmetric() if case.get("mode") == "asymmetric" else cfg


def _normal(gen, shape, std):
    return torch.randn(shape, device="cuda", generator=gen) * std


def _with_outliers(gen, rows, cols):
    """N(0,1) with 1 % of the entries fifty times larger, as the weights are that quantizers find hard."""
    w = torch.randn((rows, cols), device="cuda", generator=gen)
    w[torch.rand((rows, cols), device="cuda", generator=gen) < 0.01] *= 50.0
    return w


def _layer(gen, n, k, bias, config, std=0.02):
    b = _normal(gen, (n,), 0.1) if bias else None
    return QuantizedLinear.from_linear(Linear(_normal(gen, (n, k), std), b), config)


class _Model:
    """What quantize_named_parameters walks: named f32 weights on the device."""

    def __init__(self, params):
        self.params = params

    def named_parameters(self):
        return self.params


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind == "linear":
        cfg = _config(case)
        if case["weights"] == "int4":
            cfg = QuantConfig(QuantBits.Int4, QuantMode.Symmetric, cfg.granularity)
            qt = quantize_tensor(_normal(gen, (case["n"], case["k"]), 0.02), cfg)
            s["layer"] = QuantizedLinear.new_int4_packed(qt, _normal(gen, (case["n"],), 0.1) if case["bias"] else None)
        else:
            s["layer"] = _layer(gen, case["n"], case["k"], case["bias"], cfg)
        s["x"] = _normal(gen, (case["m"], case["k"]), 1.0).to(_DTYPE[case["x"]])
        s["epilogue"] = _lib.EPILOGUE_RELU if case["relu"] else _lib.EPILOGUE_NONE
        s["y_dtype"] = _DTYPE[case["y"]]
    elif kind == "blocks":
        cfg = QuantConfig.int8_per_channel()
        d, ff = case["d"], case["ff"]
        s["blocks"] = [(_layer(gen, ff, d, False, cfg), _layer(gen, ff, d, False, cfg), _layer(gen, d, ff, False, cfg))
                       for _ in range(case["layers"])]
        s["x"] = _normal(gen, (case["m"], d), 1.0).to(torch.bfloat16)
        if case["graph"]:
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                for _ in range(2):
                    _blocks(s)
            torch.cuda.current_stream().wait_stream(side)
            torch.cuda.synchronize()
            s["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["graph"]):
                s["y"] = _blocks(s)
    elif kind == "stack" and case["shape"] == "classifier":
        cfg = QuantConfig.int8_per_channel()
        s["layers"] = [_layer(gen, case["d_hidden"], case["d_in"], True, cfg, 0.05),
                       _layer(gen, case["d_out"], case["d_hidden"], True, cfg, 0.05)]
        s["x"] = torch.rand((case["m"], case["d_in"]), device="cuda", generator=gen)
    elif kind == "stack":
        cfg = QuantConfig.int8_per_channel()
        s["spec"] = _gpt_layers(case)
        s["layers"] = [_layer(gen, n, k, False, cfg) for n, k, _ in s["spec"]]
        s["x"] = {k: _normal(gen, (case["m"], k), 1.0) for k in (case["d"], case["ff"])}
    elif kind == "quantize":
        s["w"] = _with_outliers(gen, case["rows"], case["cols"]).to(_DTYPE[case["x"]])
        s["config"] = _config(case)
    elif kind == "model":
        s["model"] = _Model([("layer%d.weight" % i, _normal(gen, (n, k), 0.02)) for i, (n, k, _) in enumerate(_gpt_layers(case))])
        s["config"] = _config(case)
    else:
        qt = quantize_tensor(_with_outliers(gen, case["rows"], case["cols"]), _config(case))
        qt.original_dtype = _DTYPE[case["y"]]
        s["qt"] = qt
    return s


def _blocks(s):
    y = s["x"]
    for gate, up, down in s["blocks"]:
        y = down.forward(gate.forward_gate_up_silu(up, y))
    return y


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "linear":
        return s["layer"].forward(s["x"], epilogue=s["epilogue"], out_dtype=s["y_dtype"])
    if kind == "blocks":
        if case["graph"]:
            s["graph"].replay()
            return s["y"]
        return _blocks(s)
    if kind == "stack":
        if case["shape"] == "classifier":
            h = s["layers"][0].forward(s["x"], epilogue=_lib.EPILOGUE_RELU)
            return s["layers"][1].forward(h)
        return [layer.forward(s["x"][k], epilogue=_lib.EPILOGUE_RELU if relu else _lib.EPILOGUE_NONE)
                for layer, (_, k, relu) in zip(s["layers"], s["spec"])]
    if kind == "quantize":
        return _parts(quantize_tensor(s["w"], s["config"]))
    if kind == "model":
        return [_parts(qt) for _, qt in quantize_named_parameters(s["model"], s["config"])]
    return dequantize_tensor(s["qt"])


def _parts(qt):
    return [qt.data, qt.scales] + ([qt.zero_points_t] if qt.zero_points_t is not None else [])


def _forward_work(m, n, k, xs, ys, bias=False, w_bits=8):
    return n * k * w_bits // 8 + 4 * n * (2 if bias else 1) + m * k * xs + m * n * ys, 2 * m * n * k


def work(case):
    kind = case["kind"]
    parts = []
    if kind == "linear":
        parts = [_forward_work(case["m"], case["n"], case["k"], _SIZE[case["x"]], _SIZE[case["y"]], case["bias"],
                               4 if case["weights"] == "int4" else 8)]
    elif kind == "blocks":
        m, d, ff = case["m"], case["d"], case["ff"]
        # the hidden activation stays inside the block: not counted
        parts = [(3 * d * ff + 4 * (2 * ff + d) + 4 * m * d, 6 * m * d * ff)] * case["layers"]
    elif kind == "stack" and case["shape"] == "classifier":
        m = case["m"]
        parts = [(case["d_hidden"] * (case["d_in"] + 8) + case["d_out"] * (case["d_hidden"] + 8) + 4 * m * (case["d_in"] + case["d_out"]),
                  2 * m * case["d_hidden"] * (case["d_in"] + case["d_out"]))]
    elif kind == "stack":
        # (the Linears of a pass share their inputs: x of each width is read once)
        parts = [_forward_work(case["m"], n, k, 0, 4) for n, k, _ in _gpt_layers(case)] + [(4 * case["m"] * (case["d"] + case["ff"]), 0)]
    elif kind == "quantize":
        groups = case["rows"] if case["granularity"] == "channel" else 1
        parts = [(case["rows"] * case["cols"] * (_SIZE[case["x"]] + 1) + groups * (16 if case["mode"] == "asymmetric" else 8), 0)]
    elif kind == "model":
        parts = [(5 * n * k + 8 * (n if case["granularity"] == "channel" else 1), 0) for n, k, _ in _gpt_layers(case)]
    else:
        groups = case["rows"] if case["granularity"] == "channel" else 1
        parts = [(case["rows"] * case["cols"] * (_SIZE[case["y"]] + 1) + 8 * groups, 0)]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    # codes, scales and dequantized values are defined bit for bit
    if case["kind"] in ("quantize", "model", "dequantize"):
        return "exact"
    if case["kind"] == "stack" or case["kind"] == "linear" and case["x"] == "f32" and case["y"] == "f32":
        return {"rel": 1e-5}
    if case["kind"] == "linear" and case["y"] == "f32":
        return {"rel": 1e-5}  # bf16 activations and whole codes: exact products, 32-bit sums
    return {"rel": 1e-2}
