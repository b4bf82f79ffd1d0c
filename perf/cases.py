"""The work a program gives this package, as cases that can be timed and compared.

Kinds, by the public entry point that a pass calls:

  layer    BSIQuantizedLinear.forward: quantise + pack the activations, dot with the key set, cast, bias
  dot      batch_dot_product_multiquery_cuda_batch_caps on query and key capsules that are already built
  query    build_bsi_queries_cuda_batch_packed, then the dot: what the unfused layer issues per call
  queries  build_bsi_queries_cuda_batch_packed alone, all of its tensors
  keys     build_bsi_keys_cuda of one weight matrix (once per layer when a model is converted)
  encode   ewah_encode_words of bit slices;   decode   ewah_decode_words of such a stream
  opt      OPT whose linears are BSI layers (build_opt_bsi), token ids -> logits, eager
  stack    the fused decoder (build_opt_tp) on one GPU, recorded with capture(), ids -> hidden states
"""
import torch

import bsipytorch_b200
from bsipytorch_b200 import linear, opt, opt_tp

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
DECIMALS = 2


def listed():
    return [
        # one token through a 4096-wide projection: the smallest call, latency and launches
        {"name": "layer 1 token", "kind": "layer", "Q": 1, "D": 4096, "R": 4096, "dtype": "fp16", "bias": True},
        # a small decode batch through the widest layer of OPT-6.7B (fc1)
        {"name": "layer 16 tokens wide", "kind": "layer", "Q": 16, "D": 4096, "R": 16384, "dtype": "bf16", "bias": True},
        # odd sizes in float32: no power of two anywhere, depth that is no multiple of a word
        {"name": "layer ragged", "kind": "layer", "Q": 77, "D": 1000, "R": 777, "dtype": "fp32", "bias": True},
        # prefill, 16 sequences of 256 tokens through fc1 of OPT-6.7B
        {"name": "layer prefill", "kind": "layer", "Q": 4096, "D": 4096, "R": 16384, "dtype": "fp16", "bias": True},
        # the dot microbenchmark's shape (fc1 of OPT-1.3B, 512 tokens), operands prebuilt
        {"name": "dot fc1", "kind": "dot", "Q": 512, "D": 2048, "R": 8192, "dtype": "fp16", "relu": False},
        # the unfused layer's two calls on the transposed shape (fc2): deep, few output columns, relu activations
        {"name": "query fc2", "kind": "query", "Q": 512, "D": 8192, "R": 2048, "dtype": "fp16", "relu": True},
        # activations of a whole batch sliced and packed (16384 = width of fc2's input in OPT-6.7B)
        {"name": "queries batch", "kind": "queries", "Q": 4096, "D": 16384, "dtype": "fp16", "relu": False},
        # conversion of the largest weight of OPT-6.7B
        {"name": "keys fc1", "kind": "keys", "R": 16384, "D": 4096, "dtype": "fp32"},
        # slices of a batch of relu activations compressed, and such a stream expanded
        {"name": "encode slices", "kind": "encode", "rows": 4096, "W": 256, "threshold": 0.5},
        {"name": "decode slices", "kind": "decode", "rows": 4096, "W": 256, "threshold": 0.5},
        # the evaluated model at the evaluation batch (8 x 128 tokens), launch after launch from Python
        {"name": "opt-125m logits", "kind": "opt", "model": "opt-125m", "layers": 12, "B": 8, "T": 128, "dtype": "fp16"},
        # decoder layers of OPT-6.7B's widths at the serving batch (16 x 256 tokens), replayed as a graph
        {"name": "opt-6.7b stack", "kind": "stack", "model": "opt-6.7b", "layers": 4, "B": 16, "T": 256, "dtype": "fp16"},
    ]


LARGEST = 4096 * 4096 * 16384     # products in the largest dot


def _size(rng, low, high, multiple):
    """A size spread over the logarithm of [low, high]: half of the time a multiple, else any number."""
    n = int(round(low * (high / low) ** rng.random()))
    if rng.random() < 0.5:
        n = max(multiple, n // multiple * multiple)
    return max(low, min(high, n))


def _dot_sizes(rng, fewest):
    while True:
        q = _size(rng, fewest, 4096, 8)
        d, r = _size(rng, 256, 16384, 256), _size(rng, 256, 16384, 256)
        if q * d * r <= LARGEST:
            return {"Q": q, "D": d, "R": r}


def draw(rng):
    # layers are what a model issues most, so they are drawn most
    kind = rng.choice(["layer"] * 5 + ["dot", "dot", "query", "query", "queries", "keys", "encode", "decode", "opt", "stack"])
    dtype = rng.choice(["fp16", "fp16", "bf16", "fp32"])
    if kind == "layer":
        return dict(_dot_sizes(rng, 1), kind=kind, dtype=dtype, bias=rng.random() < 0.8)
    if kind in ("dot", "query"):
        return dict(_dot_sizes(rng, 16), kind=kind, dtype=dtype, relu=rng.random() < 0.4)
    if kind == "queries":
        return {"kind": kind, "Q": _size(rng, 16, 4096, 8), "D": _size(rng, 256, 16384, 256), "dtype": dtype,
                "relu": rng.random() < 0.4}
    if kind == "keys":
        return {"kind": kind, "R": _size(rng, 256, 16384, 256), "D": _size(rng, 256, 4096, 256),
                "dtype": rng.choice(["fp32", "fp32", "fp16", "bf16"])}
    if kind in ("encode", "decode"):
        return {"kind": kind, "rows": _size(rng, 16, 4096, 8), "W": _size(rng, 4, 256, 4),
                "threshold": rng.choice([0.2, 0.5])}
    if kind == "opt":
        return {"kind": kind, "model": "opt-125m", "layers": 12, "B": rng.randint(1, 8), "T": _size(rng, 16, 128, 8),
                "dtype": rng.choice(["fp16", "fp32"])}
    return {"kind": kind, "model": rng.choice(["opt-1.3b", "opt-6.7b"]), "layers": rng.randint(2, 4),
            "B": rng.randint(1, 16), "T": _size(rng, 32, 256, 32), "dtype": rng.choice(["fp16", "bf16"])}


# ---- inputs ----------------------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _activations(g, q, d, dtype, relu):
    """What a linear reads: a layer norm's output (unit variance, 1 % outliers) or a relu's (half zeros)."""
    x = torch.randn(q, d, generator=g, device="cuda")
    if relu:
        x = torch.relu(x)
    else:
        x = torch.where(torch.rand(q, d, generator=g, device="cuda") < 0.01, x * 20.0, x)
    return x.to(DTYPES[dtype])


def _weights(g, r, d):
    return torch.randn(r, d, generator=g, device="cuda") * 0.02


def _config(case):
    base = opt.CONFIGS[case["model"]]
    return opt.OPTConfig(hidden_size=base.hidden_size, num_hidden_layers=case["layers"], ffn_dim=base.ffn_dim,
                         num_attention_heads=base.num_attention_heads, name=base.name)


def _slices(g, rows, w):
    """Bit slices [rows * 7, w] of packed relu activations."""
    x = _activations(g, rows, w * 64, "fp16", True)
    caps = bsipytorch_b200.bsi_ops.build_bsi_queries_cuda_batch_packed(x, DECIMALS)
    words = bsipytorch_b200.bsi_ops.debug_query_batch_tensors(caps)["words"]
    return words.reshape(-1, words.shape[-1])


def prepare(case, seed):
    ops = bsipytorch_b200.bsi_ops
    kind, g = case["kind"], _generator(seed)
    s = {"kind": kind}
    if kind == "layer":
        lin = torch.nn.Linear(case["D"], case["R"], bias=case["bias"], device="cuda")
        with torch.no_grad():
            lin.weight.copy_(_weights(g, case["R"], case["D"]))
            if case["bias"]:
                lin.bias.copy_(torch.randn(case["R"], generator=g, device="cuda") * 0.02)
        s["layer"] = linear.BSIQuantizedLinear(lin, decimalPlaces=DECIMALS)
        s["x"] = _activations(g, case["Q"], case["D"], case["dtype"], False)
    elif kind in ("dot", "query"):
        s["keys"] = ops.build_bsi_keys_cuda(_weights(g, case["R"], case["D"]), DECIMALS)[0]
        s["x"] = _activations(g, case["Q"], case["D"], case["dtype"], case["relu"])
        if kind == "dot":
            s["queries"] = ops.build_bsi_queries_cuda_batch_packed(s["x"], DECIMALS)
    elif kind == "queries":
        s["x"] = _activations(g, case["Q"], case["D"], case["dtype"], case["relu"])
    elif kind == "keys":
        s["w"] = _weights(g, case["R"], case["D"]).to(DTYPES[case["dtype"]])
    elif kind in ("encode", "decode"):
        words = _slices(g, case["rows"], case["W"])
        if kind == "encode":
            s["words"], s["threshold"] = words, case["threshold"]
        else:
            s["stream"], s["off"], s["len"], _ = ops.ewah_encode_words(words, case["threshold"])
            s["W"] = case["W"]
    else:
        cfg = _config(case)
        s["ids"] = torch.randint(0, cfg.vocab_size, (case["B"], case["T"]), generator=g, device="cuda")
        if kind == "opt":
            s["model"] = opt.build_opt_bsi(cfg, dtype=DTYPES[case["dtype"]], seed=seed)
        else:
            s["model"] = opt_tp.build_opt_tp(cfg, dtype=DTYPES[case["dtype"]], seed=seed).capture(case["B"], case["T"])
    return s


# ---- one pass --------------------------------------------------------------------------------------------------
def _tensors(d):
    return {k: d[k] for k in ("words", "slice_weights", "scales", "q8")}


def run(s):
    ops = bsipytorch_b200.bsi_ops
    kind = s["kind"]
    if kind == "layer":
        with torch.no_grad():
            return s["layer"](s["x"])
    if kind == "dot":
        return ops.batch_dot_product_multiquery_cuda_batch_caps(s["queries"], s["keys"])[0]
    if kind == "query":
        queries = ops.build_bsi_queries_cuda_batch_packed(s["x"], DECIMALS)
        return ops.batch_dot_product_multiquery_cuda_batch_caps(queries, s["keys"])[0]
    if kind == "queries":
        return _tensors(ops.debug_query_batch_tensors(ops.build_bsi_queries_cuda_batch_packed(s["x"], DECIMALS)))
    if kind == "keys":
        return _tensors(ops.debug_keys_tensors(ops.build_bsi_keys_cuda(s["w"], DECIMALS)[0]))
    if kind == "encode":
        return ops.ewah_encode_words(s["words"], s["threshold"])
    if kind == "decode":
        return ops.ewah_decode_words(s["stream"], s["off"], s["len"], s["W"])
    with torch.no_grad():
        return s["model"](s["ids"]) if kind == "opt" else s["model"].hidden_states(s["ids"])


# ---- what a pass cannot do without -----------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    e = {"fp16": 2, "bf16": 2, "fp32": 4}.get(case.get("dtype"), 0)
    q, d, r = case.get("Q", 0), case.get("D", 0), case.get("R", 0)
    chunks, words = -(-d // 256), -(-d // 64)
    if kind == "layer":        # activations, int8 key image and row scales in; outputs out
        return {"bytes": q * d * e + r * d + 4 * r + (4 * r if case["bias"] else 0) + q * r * e, "flops": 2 * q * d * r}
    if kind == "dot":          # int8 images and scales in; float32 out
        return {"bytes": q * d + 4 * q * chunks + r * d + 4 * r + 4 * q * r, "flops": 2 * q * d * r}
    if kind == "query":        # the query capsule (7 slices, int8 image, scales) is written as well
        built = 7 * q * (8 * words + 4) + q * 256 * chunks + 4 * q * chunks
        return {"bytes": q * d * e + built + r * d + 4 * r + 4 * q * r, "flops": 2 * q * d * r}
    if kind == "queries":
        return {"bytes": q * d * e + 7 * q * (8 * words + 4) + q * 256 * chunks + 4 * q * chunks, "flops": 0}
    if kind == "keys":         # 6 slices and their weights, int8 image, row scales
        return {"bytes": r * d * e + 6 * r * (8 * words + 4) + r * 256 * chunks + 4 * r, "flops": 0}
    if kind in ("encode", "decode"):   # about as many words in the stream as in the slices
        return {"bytes": 2 * 8 * 7 * case["rows"] * case["W"], "flops": 0}
    cfg = _config(case)
    h, f, n = cfg.hidden_size, cfg.ffn_dim, case["B"] * case["T"]
    per_layer = 4 * h * h + 2 * h * f
    flops = case["layers"] * (2 * n * per_layer + 2 * n * case["T"] * h)     # causal: half of the score matrix
    size = case["layers"] * per_layer + 8 * n
    if kind == "opt":
        return {"bytes": size + cfg.vocab_size * (h + n) * e, "flops": flops + 2 * n * h * cfg.vocab_size}
    return {"bytes": size + n * h * 3 * e, "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind in ("queries", "keys", "encode", "decode"):
        return "exact"         # integers, words, powers of two
    if kind in ("opt", "stack"):
        # one last bit of an activation becomes a whole step where it is quantised again
        return {"rel": 1e-2, "max": 0.2}
    if case.get("dtype") == "fp16" and kind == "layer":
        return {"rel": 5e-4, "max": 2e-3}      # one rounding to 11 bits
    if case.get("dtype") == "bf16" and kind == "layer":
        return {"rel": 4e-3, "max": 1.6e-2}    # one rounding to 8 bits
    return {"rel": 1e-6, "max": 1e-5}          # float32 sums of exact integers over at most 64 chunks
