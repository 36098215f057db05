"""The work this library is timed on: whole transformer blocks through compile_model() and
Model.run_with_tensors(), and the eager kernels of aitemplate_b200.kernels, over the sizes, data types and options
that inference programs call them with. (There is no training here: the library runs forward passes only.)

listed() names a fixed set, draw() gives more of the same ranges; prepare() makes what a program holds before the call,
run() is one call, work() what it cannot do without, tolerance() how far two correct results may lie apart, exact()
what the call returns when all of it is computed in 64 bits.
"""
from __future__ import annotations

import math
import tempfile

import torch
import torch.nn.functional as F

from aitemplate_b200 import kernels
from aitemplate_b200.compiler import compile_model
from aitemplate_b200.testing import detect_target, workloads

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
_HIDDEN, _FFN = 768, 3072
_SD = workloads.SD_BLOCK
_RESIDUAL = ("add", "add_relu", "mul")


def listed():
    return [
        # one request, answered as soon as it can be: encoder layer at batch 1, the call's default synchronous form
        {"name": "bert_b1_s384", "kind": "bert", "batch": 1, "seq": 384, "graph": True, "sync": True},
        # a few requests of an odd length, every argument of the call at its default (eager, synchronous)
        {"name": "bert_b5_s211_eager", "kind": "bert", "batch": 5, "seq": 211, "graph": False, "sync": True},
        # offline throughput, the batch and length the BERT benchmark is quoted on
        {"name": "bert_b64_s384", "kind": "bert", "batch": 64, "seq": 384, "graph": True, "sync": False},
        # long documents: most of the time is attention
        {"name": "bert_b4_s4096", "kind": "bert", "batch": 4, "seq": 4096, "graph": True, "sync": False},
        # one UNet transformer block of an image pipeline, 64 x 64 latents, conditional + unconditional in one batch
        {"name": "sd_b2_t4096", "kind": "sd", "batch": 2, "tokens": 4096, "graph": True, "sync": False},
        # one token of a decoder: a matrix-vector product against a large weight
        {"name": "gemm_m1_8192", "kind": "gemm", "m": 1, "n": 8192, "k": 8192, "dtype": "fp16", "epilogue": "relu"},
        # first feed-forward projection of a short batch: a call of a few microseconds
        {"name": "gemm_256x3072x768_gelu", "kind": "gemm", "m": 256, "n": 3072, "k": 768, "dtype": "fp16",
         "epilogue": "fast_gelu"},
        # a prompt of 1000 tokens through a projection with its residual
        {"name": "gemm_1000x4096_bf16_add", "kind": "gemm", "m": 1000, "n": 4096, "k": 4096, "dtype": "bf16",
         "epilogue": "add"},
        # a large dense layer: the rate of the tensor cores
        {"name": "gemm_8192_relu", "kind": "gemm", "m": 8192, "n": 8192, "k": 8192, "dtype": "fp16", "epilogue": "relu"},
        # causal prefill of eight packed sequences of different lengths, the longest 4096 tokens
        {"name": "flash_bf16_d128_causal", "kind": "attention", "packed": True, "seqs": 8, "longest": 4096, "heads": 16,
         "dim": 128, "dtype": "bf16", "causal": True},
        # attention scores of many heads as a batched product
        {"name": "bmm_rcr_1024x512x64", "kind": "bmm", "batch": 1024, "m": 512, "n": 512, "k": 64, "dtype": "fp16",
         "b_row_major": False},
        # the memory-bound operators over the activations of a batch
        {"name": "rowwise_64x384x1024", "kind": "rowwise", "batch": 64, "seq": 384, "n": 1024, "dtype": "fp16"},
    ]


def _log_int(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, round(v / step) * step)))


def draw(rng):
    kind = rng.choice(("bert", "bert", "sd", "gemm", "gemm", "gemm", "attention", "bmm", "rowwise"))
    dtype = rng.choice(("fp16", "bf16"))
    if kind == "bert":
        while True:
            # token counts of every kind: padded to a multiple of 32 by some callers, as they come by others
            batch, seq = _log_int(rng, 1, 64), _log_int(rng, 32, 4096, rng.choice((1, 32)))
            if batch * seq <= 24576 and workloads.bert_layer_flops(batch, seq) <= 4.6e11:
                break
        graph = rng.random() < 0.7
        return {"kind": kind, "batch": batch, "seq": seq, "graph": graph, "sync": batch * seq < 4096}
    if kind == "sd":
        # latents of h x w with sides in multiples of 8
        tokens = 8 * rng.randint(2, 8) * 8 * rng.randint(2, 8)
        return {"kind": kind, "batch": rng.choice((1, 2, 4) if tokens <= 2048 else (1, 2)), "tokens": tokens,
                "graph": True, "sync": False}
    if kind == "gemm":
        while True:
            # N of any value (a vocabulary), K a whole number of 16-byte vectors
            m = _log_int(rng, 1, 8192)
            n = _log_int(rng, 256, 8192, rng.choice((1, 8, 64, 64)))
            k = _log_int(rng, 256, 8192, rng.choice((8, 64, 64)))
            if 2.0 * m * n * k <= 1.1e12:
                break
        epilogue = rng.choice(("", "", "relu", "gelu", "fast_gelu", "tanh", "add", "add", "add_relu", "mul"))
        return {"kind": kind, "m": m, "n": n, "k": k, "dtype": dtype, "epilogue": epilogue}
    if kind == "attention":
        longest = _log_int(rng, 64, 4096)
        seqs = rng.randint(1, 8)
        return {"kind": kind, "packed": rng.random() < 0.5, "seqs": seqs, "longest": longest,
                "heads": rng.choice((8, 12, 16)), "dim": rng.choice((40, 64, 64, 80, 128)), "dtype": dtype,
                "causal": rng.random() < 0.5}
    if kind == "bmm":
        return {"kind": kind, "batch": _log_int(rng, 16, 1024), "m": _log_int(rng, 64, 512), "n": _log_int(rng, 64, 512, 8),
                "k": _log_int(rng, 32, 128, 8), "dtype": dtype, "b_row_major": rng.random() < 0.3}
    return {"kind": kind, "batch": _log_int(rng, 1, 64), "seq": _log_int(rng, 64, 384),
            "n": _log_int(rng, 64, 1024, rng.choice((1, 8, 64))), "dtype": dtype}


# ------------------------------------------------------------------------------------------------ what a program holds


def _lengths(case):
    """Sequence lengths of an attention case: spread evenly from longest / seqs to longest."""
    return [max(1, case["longest"] * (i + 1) // case["seqs"]) for i in range(case["seqs"])]


def _model(output, name):
    with tempfile.TemporaryDirectory() as workdir:
        return compile_model(output, detect_target(), workdir, name)


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    dtype = _DTYPES[case.get("dtype", "fp16")]

    def normal(*shape, scale=1.0):
        return torch.randn(shape, generator=gen, device="cuda").mul_(scale).to(dtype)

    def uniform(*shape, lo=-1.0, hi=1.0):
        return torch.rand(shape, generator=gen, device="cuda").mul_(hi - lo).add_(lo).to(dtype)

    if kind == "bert":
        batch, seq = case["batch"], case["seq"]
        params = {"qkv_weight": normal(3 * _HIDDEN, _HIDDEN, scale=0.02), "qkv_bias": normal(3 * _HIDDEN, scale=0.02),
                  "proj_weight": normal(_HIDDEN, _HIDDEN, scale=0.02), "proj_bias": normal(_HIDDEN, scale=0.02),
                  "fc1_weight": normal(_FFN, _HIDDEN, scale=0.02), "fc1_bias": normal(_FFN, scale=0.02),
                  "fc2_weight": normal(_HIDDEN, _FFN, scale=0.02), "fc2_bias": normal(_HIDDEN, scale=0.02)}
        for ln in ("ln1", "ln2"):
            params[ln + "_gamma"] = uniform(_HIDDEN, lo=0.5, hi=1.5)
            params[ln + "_beta"] = normal(_HIDDEN, scale=0.1)
        return {"params": params, "inputs": {"hidden_states": normal(batch, seq, _HIDDEN)}}
    if kind == "sd":
        batch, tokens, dim = case["batch"], case["tokens"], _SD["dim"]
        params = {}
        for name, cdim in (("attn1", dim), ("attn2", _SD["context_dim"])):
            params[f"{name}_to_q_weight"] = normal(dim, dim, scale=0.02)
            params[f"{name}_to_k_weight"] = normal(dim, cdim, scale=0.02)
            params[f"{name}_to_v_weight"] = normal(dim, cdim, scale=0.02)
            params[f"{name}_to_out_weight"] = normal(dim, dim, scale=0.02)
            params[f"{name}_to_out_bias"] = normal(dim, scale=0.02)
        for name in ("norm1", "norm2", "norm3"):
            params[f"{name}_weight"] = uniform(dim, lo=0.5, hi=1.5)
            params[f"{name}_bias"] = normal(dim, scale=0.1)
        for name in ("ff_proj", "ff_gate"):
            params[f"{name}_weight"] = normal(4 * dim, dim, scale=0.02)
            params[f"{name}_bias"] = normal(4 * dim, scale=0.02)
        params["ff_out_weight"] = normal(dim, 4 * dim, scale=0.02)
        params["ff_out_bias"] = normal(dim, scale=0.02)
        return {"params": params, "inputs": {"latent": normal(batch, tokens, dim),
                                             "context": normal(batch, _SD["context_tokens"], _SD["context_dim"])}}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"x": uniform(m, k), "w": normal(n, k, scale=0.01), "bias": normal(n, scale=0.01),
                "d0": normal(m, n) if case["epilogue"] in _RESIDUAL else None}
    if kind == "attention":
        lengths, heads, dim = _lengths(case), case["heads"], case["dim"]
        if case["packed"]:
            starts = torch.tensor([0] + lengths, device="cuda").cumsum(0).to(torch.int32)
            return {"qkv": normal(sum(lengths), 3, heads, dim), "cu_seqlens": starts}
        q, k, v = (normal(case["seqs"], heads, case["longest"], dim) for _ in range(3))
        return {"q": q, "k": k, "v": v,
                "lengths_kv": torch.tensor(lengths, dtype=torch.int32, device="cuda")}
    if kind == "bmm":
        batch, m, n, k = case["batch"], case["m"], case["n"], case["k"]
        return {"a": uniform(batch, m, k),
                "b": uniform(batch, k, n) if case["b_row_major"] else uniform(batch, n, k)}
    n = case["n"]
    return {"x": normal(case["batch"], case["seq"], n, scale=2.0), "gamma": uniform(n, lo=0.5, hi=1.5),
            "beta": normal(n, scale=0.1)}


def prepare(case, seed):
    state = {"case": case, **_inputs(case, seed)}
    if case["kind"] == "bert":
        _, y = workloads.build_bert_layer(case["batch"], case["seq"])
        state["model"] = _model(y, "bert_layer")
        state["model"].set_many_constants_with_tensors(
            {n: state["params"][k] for n, k in workloads.BERT_PARAM_NAMES.items()})
        state["outputs"] = {"output_0": torch.empty_like(state["inputs"]["hidden_states"])}
    elif case["kind"] == "sd":
        state["model"] = _model(workloads.build_sd_block(case["batch"], tokens=case["tokens"]), "sd_block")
        state["model"].set_many_constants_with_tensors(state["params"])
        state["outputs"] = {"output_0": torch.empty_like(state["inputs"]["latent"])}
    return state


# ------------------------------------------------------------------------------------------------------------ one call


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("bert", "sd"):
        return state["model"].run_with_tensors(state["inputs"], state["outputs"], sync=case["sync"],
                                               graph_mode=case["graph"])
    if kind == "gemm":
        return kernels.gemm_rcr(state["x"], state["w"], state["bias"], state["d0"], epilogue=case["epilogue"])
    if kind == "attention":
        if case["packed"]:
            return kernels.flash_attention(state["qkv"], state["cu_seqlens"], case["longest"], causal=case["causal"])
        return kernels.mem_eff_attention(state["q"], state["k"], state["v"], causal=case["causal"],
                                         lengths_kv=state["lengths_kv"])
    if kind == "bmm":
        return (kernels.bmm_rrr if case["b_row_major"] else kernels.bmm_rcr)(state["a"], state["b"])
    x = state["x"]
    parts = kernels.split(x, (case["n"] + 3) // 4, dim=2)
    return {"layernorm": kernels.layernorm(x, state["gamma"], state["beta"]), "softmax": kernels.softmax(x),
            "parts": parts, "joined": kernels.concatenate(parts[::-1], dim=2), "turned": kernels.permute(x, (0, 2, 1))}


# ---------------------------------------------------------------------------------------------------- what it amounts to


def work(case):
    kind = case["kind"]
    if kind == "bert":
        rows = case["batch"] * case["seq"]
        weights = 4 * _HIDDEN * _HIDDEN + 2 * _HIDDEN * _FFN + 3 * _HIDDEN + _HIDDEN + _FFN + _HIDDEN + 4 * _HIDDEN
        return {"bytes": 2 * (2 * rows * _HIDDEN + weights),
                "flops": workloads.bert_layer_flops(case["batch"], case["seq"])}
    if kind == "sd":
        batch, tokens, dim = case["batch"], case["tokens"], _SD["dim"]
        rows, ctx_rows, ctx = batch * tokens, batch * _SD["context_tokens"], _SD["context_dim"]
        weights = 6 * dim * dim + 2 * dim * ctx + 12 * dim * dim
        gemms = 2.0 * rows * dim * dim * (4 + 2 + 8 + 4) + 2.0 * ctx_rows * ctx * dim * 2
        attn = 4.0 * rows * dim * (tokens + _SD["context_tokens"])
        return {"bytes": 2 * (2 * rows * dim + ctx_rows * ctx + weights), "flops": gemms + attn}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        residual = m * n if case["epilogue"] in _RESIDUAL else 0
        return {"bytes": 2 * (m * k + n * k + n + m * n + residual), "flops": 2.0 * m * n * k}
    if kind == "attention":
        lengths, heads, dim, longest = _lengths(case), case["heads"], case["dim"], case["longest"]
        pairs = 0
        for length in lengths:
            rows = length if case["packed"] else longest
            if case["causal"]:  # row i sees the keys up to i, and none past the sequence's length
                pairs += length * (length + 1) // 2 + (rows - length) * length
            else:
                pairs += rows * length
        if case["packed"]:
            values = 4 * sum(lengths)
        else:
            values = 2 * case["seqs"] * longest + 2 * sum(lengths)
        return {"bytes": 2 * values * heads * dim, "flops": 4.0 * pairs * heads * dim}
    if kind == "bmm":
        batch, m, n, k = case["batch"], case["m"], case["n"], case["k"]
        return {"bytes": 2 * batch * (m * k + n * k + m * n), "flops": 2.0 * batch * m * n * k}
    values = case["batch"] * case["seq"] * case["n"]
    return {"bytes": 5 * 2 * 2 * values, "flops": 20.0 * values}


def tolerance(case):
    # about four times what the paths show against the same expressions in 64 bits on the GPU (fp16: a whole encoder
    # layer 4.2e-4 and 2.4e-3, one product 2.1e-4 and 5e-4; bf16: attention 2.3e-3 and 3.4e-2, one product 1.7e-3 and 4e-3)
    half = case.get("dtype", "fp16") == "fp16"
    return {"rel": 1.7e-3 if half else 9e-3, "max": 1e-2 if half else 0.14}


# --------------------------------------------------------------------------------------- the same expressions in 64 bits


def _attend(q, k, v, causal=False, length=None):
    """softmax(q k^T / sqrt(d)) v of one sequence, [heads, rows, d] -> [rows, heads, d], 1024 query rows at a time."""
    out, keys = [], torch.arange(k.shape[1], device=q.device)
    for r0 in range(0, q.shape[1], 1024):
        s = q[:, r0:r0 + 1024] @ k.transpose(1, 2) / math.sqrt(q.shape[2])
        if length is not None:
            s = s.masked_fill(keys >= length, -math.inf)
        if causal:
            rows = torch.arange(r0, r0 + s.shape[1], device=q.device)
            s = s.masked_fill(keys > rows[:, None], -math.inf)
        out.append((torch.softmax(s, dim=-1) @ v).transpose(0, 1))
    return torch.cat(out)


def _heads(x, heads):
    return x.reshape(x.shape[0], heads, -1).transpose(0, 1)


def _encoder_layer(x, p):
    def one(h):  # [seq, hidden]
        q, k, v = (_heads(t, 12) for t in F.linear(h, p["qkv_weight"], p["qkv_bias"]).chunk(3, dim=1))
        a = F.linear(_attend(q, k, v).reshape(h.shape), p["proj_weight"], p["proj_bias"]) + h
        a = F.layer_norm(a, a.shape[1:], p["ln1_gamma"], p["ln1_beta"], workloads.BERT_BASE["eps"])
        f = F.gelu(F.linear(a, p["fc1_weight"], p["fc1_bias"]), approximate="tanh")
        f = F.linear(f, p["fc2_weight"], p["fc2_bias"]) + a
        return F.layer_norm(f, f.shape[1:], p["ln2_gamma"], p["ln2_beta"], workloads.BERT_BASE["eps"])

    return torch.stack([one(h) for h in x])


def _unet_block(x, context, p):
    def norm(name, t):
        return F.layer_norm(t, t.shape[1:], p[name + "_weight"], p[name + "_bias"], _SD["eps"])

    def attention(name, h, ctx):
        q, k, v = (_heads(F.linear(t, p[f"{name}_to_{n}_weight"]), _SD["heads"]) for n, t in (("q", h), ("k", ctx), ("v", ctx)))
        return F.linear(_attend(q, k, v).reshape(h.shape), p[name + "_to_out_weight"], p[name + "_to_out_bias"])

    def one(t, ctx):
        h = norm("norm1", t)
        t = t + attention("attn1", h, h)
        t = t + attention("attn2", norm("norm2", t), ctx)
        h = norm("norm3", t)
        gate = F.gelu(F.linear(h, p["ff_gate_weight"], p["ff_gate_bias"]), approximate="tanh")
        h = F.linear(h, p["ff_proj_weight"], p["ff_proj_bias"]) * gate
        return t + F.linear(h, p["ff_out_weight"], p["ff_out_bias"])

    return torch.stack([one(*pair) for pair in zip(x, context)])


def exact(case, seed):
    def wide(v):
        if isinstance(v, dict):
            return {name: wide(t) for name, t in v.items()}
        return v.double() if torch.is_tensor(v) and v.is_floating_point() else v

    given, kind = wide(_inputs(case, seed)), case["kind"]
    if kind == "bert":
        return {"output_0": _encoder_layer(given["inputs"]["hidden_states"], given["params"])}
    if kind == "sd":
        return {"output_0": _unet_block(given["inputs"]["latent"], given["inputs"]["context"], given["params"])}
    if kind == "gemm":
        y, d0 = F.linear(given["x"], given["w"], given["bias"]), given["d0"]
        return {"": lambda: y, "relu": lambda: torch.relu(y), "gelu": lambda: F.gelu(y), "tanh": lambda: torch.tanh(y),
                "fast_gelu": lambda: F.gelu(y, approximate="tanh"), "add": lambda: y + d0,
                "add_relu": lambda: torch.relu(y + d0), "mul": lambda: y * d0}[case["epilogue"]]()
    if kind == "attention":
        causal, lengths = case["causal"], _lengths(case)
        if case["packed"]:
            return torch.cat([_attend(*t.permute(1, 2, 0, 3), causal) for t in given["qkv"].split(lengths)])
        return torch.stack([_attend(q, k, v, causal, length)
                            for q, k, v, length in zip(given["q"], given["k"], given["v"], lengths)])
    if kind == "bmm":
        return given["a"] @ (given["b"] if case["b_row_major"] else given["b"].transpose(1, 2))
    x, n = given["x"], case["n"]
    parts = list(x.split((n + 3) // 4, dim=2))
    return {"layernorm": F.layer_norm(x, (n,), given["gamma"], given["beta"], 1e-5), "softmax": torch.softmax(x, dim=-1),
            "parts": parts, "joined": torch.cat(parts[::-1], dim=2), "turned": x.transpose(1, 2)}
