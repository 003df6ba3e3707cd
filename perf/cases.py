"""Work that a program built on this library gives it, as cases that can be timed and compared.

Three groups.  The products and attentions of a prompt portion (512 positions or fewer, the most one batched pass takes)
at the widths of the `.yalm` architectures; the one-token ops of a decode step; whole calls through Model /
InferenceState.  The layered architectures add windowed attention over a bf16 ring and the matrix-state recurrence.
Every case goes through include/yalm_b200.h (device pointers of torch tensors) or yalm_b200.api.

Inputs have the scales that the path meets: normalised activations (about 1), weights of 1 / sqrt(fan-in), unit keys for
the delta rule, decays just below 1."""
import ctypes as C
import math

import numpy as np
import torch

from yalm_b200 import api
from yalm_b200 import yalm_file as yf

DTYPES = {"fp32": (torch.float32, api.F32, 4), "fp16": (torch.float16, api.F16, 2), "bf16": (torch.bfloat16, api.BF16, 2), "fp8": (torch.uint8, api.F8E4M3, 1)}


def listed():
    return [
        # a short message: the attention-output product of a 4096-wide layer over 17 positions, added to the residual stream
        {"name": "gemm_short_prompt", "kind": "gemm", "M": 17, "N": 4096, "K": 4096, "dtype": "fp16", "accumulate": True},
        # a full prompt portion through the down projection of the 4096-wide feed-forward
        {"name": "gemm_down_portion", "kind": "gemm", "M": 512, "N": 4096, "K": 14336, "dtype": "fp16", "accumulate": True},
        # the same portion through the fused gate and up projection
        {"name": "glu_portion", "kind": "glu", "M": 512, "N": 14336, "K": 4096, "act": "silu"},
        # causal attention of the first portion of a prompt ...
        {"name": "attention_first_portion", "kind": "prompt_attention", "n": 512, "pos0": 0, "heads": 32, "kv_heads": 8, "head_dim": 128},
        # ... and of the last, ragged portion of an 8k prompt
        {"name": "attention_late_portion", "kind": "prompt_attention", "n": 507, "pos0": 7680, "heads": 32, "kv_heads": 8, "head_dim": 128},
        # a layered model's portion: window 1024 and pooled blocks of 64 behind it, bf16 ring
        {"name": "window_attention_portion", "kind": "window_attention", "n": 512, "pos0": 3584, "heads": 16, "kv_heads": 4, "dk": 128, "dv": 128,
         "window": 1024, "pool": 64},
        # a layered model's portion through the gated delta rule with a decay per key channel, the state carried over
        {"name": "delta_rule_portion", "kind": "scan", "form": "delta_channel", "n": 512, "pos0": 512, "heads": 16, "D": 128, "P": 128},
        # one decoded token's attention: early in a conversation, and at 4096 positions
        {"name": "decode_attention_early", "kind": "decode_attention", "kv_len": 37, "heads": 32, "kv_heads": 8, "head_dim": 128},
        {"name": "decode_attention_4k", "kind": "decode_attention", "kv_len": 4096, "heads": 32, "kv_heads": 8, "head_dim": 128},
        # one decoded token's feed-forward (norm, gate and up, activation, down, residual)
        {"name": "decode_ffn", "kind": "decode_ffn", "dim": 4096, "hidden": 14336, "dtype": "fp16", "act": "silu"},
        # whole calls on four layers of the 4096-wide architecture: one decoded token at 4096 positions, and a scored prompt portion
        {"name": "model_decode_4k", "kind": "model_decode", "dim": 4096, "hidden": 14336, "head_dim": 128, "heads": 32, "kv_heads": 8, "layers": 4,
         "vocab": 32000, "context": 4096},
        {"name": "model_prompt_portion", "kind": "model_prompt", "dim": 4096, "hidden": 14336, "head_dim": 128, "heads": 32, "kv_heads": 8, "layers": 4,
         "vocab": 32000, "n": 512},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "glu", "prompt_attention", "prompt_attention", "window_attention", "scan", "decode_attention", "decode_attention",
                       "decode_ffn", "model_decode", "model_prompt"])
    if kind == "gemm":
        return {"kind": kind, "M": _log(rng, 1, 512), "N": 4 * _log(rng, 128, 4096), "K": 8 * _log(rng, 64, 1792), "dtype": rng.choice(["fp16", "bf16"]),
                "accumulate": rng.random() < 0.5}
    if kind == "glu":
        return {"kind": kind, "M": _log(rng, 1, 512), "N": 8 * _log(rng, 128, 1792), "K": 8 * _log(rng, 64, 512), "act": rng.choice(["silu", "gelu"])}
    if kind in ("prompt_attention", "decode_attention"):
        heads, kv, hd = rng.choice([(32, 8, 128), (32, 8, 64), (16, 4, 128), (8, 2, 128), (16, 8, 32), (8, 8, 128), (64, 8, 128)])
        if kind == "decode_attention":
            return {"kind": kind, "kv_len": _log(rng, 1, 32768), "heads": heads, "kv_heads": kv, "head_dim": hd}
        return {"kind": kind, "n": _log(rng, 2, 512), "pos0": rng.choice([0, _log(rng, 32, 7680)]), "heads": heads, "kv_heads": kv, "head_dim": hd}
    if kind == "window_attention":
        heads, kv = rng.choice([(16, 4), (8, 2), (32, 8), (16, 16)])
        dk, dv = rng.choice([(128, 128), (64, 64), (64, 128), (128, 64)])
        return {"kind": kind, "n": _log(rng, 32, 512), "pos0": rng.choice([0, _log(rng, 64, 3584)]), "heads": heads, "kv_heads": kv, "dk": dk, "dv": dv,
                "window": rng.choice([128, 500, 1024, 2048]), "pool": rng.choice([0, 64])}
    if kind == "scan":
        D, P = rng.choice([(128, 128), (64, 64), (128, 64), (64, 128)])
        return {"kind": kind, "form": rng.choice(["delta_channel", "delta_head", "linear_channel"]), "n": _log(rng, 1, 512), "pos0": rng.choice([0, 512]),
                "heads": rng.choice([4, 8, 16]), "D": D, "P": P}
    if kind == "decode_ffn":
        return {"kind": kind, "dim": 64 * _log(rng, 16, 64), "hidden": 64 * _log(rng, 32, 224), "dtype": rng.choice(["fp16", "fp8", "fp32"]),
                "act": rng.choice(["silu", "gelu"])}
    dim, hidden, hd, heads, kv = rng.choice([(4096, 14336, 128, 32, 8), (2048, 8192, 64, 32, 8), (1024, 2816, 128, 8, 2)])
    case = {"kind": kind, "dim": dim, "hidden": hidden, "head_dim": hd, "heads": heads, "kv_heads": kv, "layers": rng.choice([2, 3]), "vocab": 32000}
    if kind == "model_decode":
        return dict(case, context=_log(rng, 16, 4096))
    return dict(case, n=_log(rng, 16, 512))


# ---- inputs ------------------------------------------------------------------------------------------------------------
def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + salt)
    return g


def _normal(g, shape, std=1.0, dtype=torch.float32):
    return (torch.randn(shape, generator=g, device="cuda", dtype=torch.float32) * std).to(dtype)


def _uniform(g, shape, lo, hi):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float32) * (hi - lo) + lo


def _weight(g, rows, cols, dtype):
    """A (rows, cols) matrix of 1 / sqrt(cols): as stored, and its row scales (fp8 only)."""
    w = _normal(g, (rows, cols), cols ** -0.5)
    if dtype != "fp8":
        return w.to(DTYPES[dtype][0]), None
    scale = (w.abs().amax(dim=1) / 448.0).clamp_min(1e-30)
    return (w / scale[:, None]).to(torch.float8_e4m3fn).view(torch.uint8), scale


def _plain(w, scale):
    """The matrix in 64 bits."""
    if scale is None:
        return w.double()
    return w.view(torch.float8_e4m3fn).float().double() * scale.double()[:, None]


def _inputs(c, seed):
    """The tensors of a case's call, from the seed alone."""
    kind = c["kind"]
    if kind in ("gemm", "glu"):
        g = _gen(seed, 1)
        dt = DTYPES[c.get("dtype", "fp16")][0]
        t = {"a": _normal(g, (c["M"], c["K"]), 1.0, dt), "w": _normal(g, (c["N"], c["K"]), c["K"] ** -0.5, dt)}
        if kind == "glu":
            t["w3"] = _normal(g, (c["N"], c["K"]), c["K"] ** -0.5, dt)
        else:
            t["c"] = _normal(g, (c["M"], c["N"])) if c["accumulate"] else torch.zeros((c["M"], c["N"]), device="cuda")
        return t
    if kind in ("prompt_attention", "decode_attention"):
        g = _gen(seed, 2)
        rows = c["kv_len"] if kind == "decode_attention" else c["pos0"] + c["n"]
        ring = (rows + 255) // 256 * 256
        nq = 1 if kind == "decode_attention" else c["n"]
        t = {"k": _normal(g, (c["kv_heads"], ring, c["head_dim"]), 1.0, torch.float16), "v": _normal(g, (c["kv_heads"], ring, c["head_dim"]), 1.0, torch.float16)}
        t["q"] = _normal(g, (nq, c["heads"], c["head_dim"]), 1.0, torch.float32 if kind == "decode_attention" else torch.float16)
        return t
    if kind == "window_attention":
        g = _gen(seed, 3)
        ring = (c["window"] + 512 + 63) // 64 * 64  # the window and the longest portion
        blocks = max(1, (c["pos0"] + c["n"]) // max(1, c["pool"]))
        t = {"k": _normal(g, (c["kv_heads"], ring, c["dk"]), 1.0, torch.bfloat16), "v": _normal(g, (c["kv_heads"], ring, c["dv"]), 1.0, torch.bfloat16)}
        t["q"] = _normal(g, (c["n"], c["heads"], c["dk"]))
        if c["pool"]:
            t["kp"] = _normal(g, (c["kv_heads"], blocks, c["dk"]), c["pool"] ** -0.5)
            t["vp"] = _normal(g, (c["kv_heads"], blocks, c["dv"]), c["pool"] ** -0.5)
        return t
    if kind == "scan":
        g = _gen(seed, 4)
        n, H, D, P = c["n"], c["heads"], c["D"], c["P"]
        k, q = _normal(g, (n, H, D)), _normal(g, (n, H, D))
        t = {"k": k / k.norm(dim=-1, keepdim=True), "q": q / q.norm(dim=-1, keepdim=True) * D ** -0.5, "v": _normal(g, (n, H, P))}
        shape = (n, H) if c["form"] == "delta_head" else (n, H, D)
        t["decay"] = torch.exp(-_uniform(g, shape, 0.0, 0.2) * _uniform(g, shape, 0.0, 1.0))
        if c["form"] != "linear_channel":
            t["beta"] = torch.sigmoid(_normal(g, (n, H)))
        t["state"] = _normal(g, (H, P, D), 0.3)
        return t
    if kind == "decode_ffn":
        g = _gen(seed, 5)
        t = {"x": _normal(g, (c["dim"],)), "norm": 1.0 + 0.1 * _normal(g, (c["dim"],))}
        for name, rows, cols in (("w1", c["hidden"], c["dim"]), ("w3", c["hidden"], c["dim"]), ("w2", c["dim"], c["hidden"])):
            t[name], t["s" + name[1:]] = _weight(g, rows, cols, c["dtype"])
        return t
    raise ValueError(kind)


def _arch(c):
    rows = c["context"] + 1 if c["kind"] == "model_decode" else c["n"]
    return yf.Arch(c["dim"], c["hidden"], c["head_dim"], c["layers"], c["heads"], c["kv_heads"], c["vocab"], (rows + 255) // 256 * 256, 1000000.0)


def _model_tensors(c, seed):
    """(name, tensor) of the model's checkpoint: embedding of 1, weights of 1 / sqrt(fan-in), a head of 4 / sqrt(dim), norms about 1."""
    q, kv, d, h = c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"], c["dim"], c["hidden"]
    plan = [("model.embed.weight", (c["vocab"], d), 1.0)]
    for l in range(c["layers"]):
        p = "model.layers.%d." % l
        plan += [(p + "attn.norm.weight", (d,), 0.0), (p + "attn.wq.weight", (q, d), d ** -0.5), (p + "attn.wk.weight", (kv, d), d ** -0.5),
                 (p + "attn.wv.weight", (kv, d), d ** -0.5), (p + "attn.wo.weight", (d, q), q ** -0.5), (p + "mlp.norm.weight", (d,), 0.0),
                 (p + "mlp.w1.weight", (h, d), d ** -0.5), (p + "mlp.w2.weight", (d, h), h ** -0.5), (p + "mlp.w3.weight", (h, d), d ** -0.5)]
    plan += [("model.norm.weight", (d,), 0.0), ("model.output.weight", (c["vocab"], d), 4.0 * d ** -0.5)]
    for i, (name, shape, std) in enumerate(plan):
        g = _gen(seed, 100 + i)
        yield name, 1.0 + 0.1 * _normal(g, shape) if std == 0.0 else _normal(g, shape, std, torch.float16)


def _tokens(c, seed):
    """The prompt, and the token that each position is scored on."""
    n = c["context"] + 1 if c["kind"] == "model_decode" else c["n"]
    ids = np.random.default_rng([seed, 6]).integers(3, c["vocab"], n + 1).astype(np.int32)
    ids[0] = 1
    return ids[:-1], ids[1:]


# ---- calls --------------------------------------------------------------------------------------------------------------
def _arg(v):
    if v is None:
        return C.c_void_p(None)
    if isinstance(v, torch.Tensor):
        return C.c_void_p(v.data_ptr())
    return C.c_float(v) if isinstance(v, float) else C.c_int(v)


def _call(name, *args):
    """The entry point with its arguments laid out once, as a program that calls it in a loop does."""
    return getattr(api.lib(), name), [_arg(v) for v in args] + [C.c_void_p(None)]


def prepare(case, seed):
    c = case
    if c["kind"] in ("model_decode", "model_prompt"):
        arch = _arch(c)
        tensors = {name: t.cpu().numpy() for name, t in _model_tensors(c, seed)}
        tensors["tokenizer.tokens"] = yf.synthetic_tokens(c["vocab"])
        model = api.Model(yf.build_image(tensors, yf.metadata_of(arch, "fp16"))).cuda()
        del tensors
        state = api.InferenceState(model)
        ids, targets = _tokens(c, seed)
        if c["kind"] == "model_decode":
            step = model.batch_capacity()
            for at in range(0, c["context"], step):
                state.forward_batch(ids[at: min(at + step, c["context"])], at)
        return {"kind": c["kind"], "state": state, "model": model, "ids": ids, "targets": targets, "pos": c.get("context", 0)}
    t = _inputs(c, seed)
    s = {"keep": t, "calls": []}
    if c["kind"] == "gemm":
        M, N, K = c["M"], c["N"], c["K"]
        if c["dtype"] == "fp16":
            s["calls"].append(_call("yalm_gemm_f16", t["c"], N, t["a"], t["w"], M, N, K, int(c["accumulate"])))
        else:
            s["calls"].append(_call("yalm_gemm_16", t["c"], N, t["a"], t["w"], M, N, K, int(c["accumulate"]), 1, 1.0))
        s["out"] = t["c"]
    elif c["kind"] == "glu":
        out = torch.empty((c["M"], c["N"]), device="cuda", dtype=torch.float16)
        s["calls"].append(_call("yalm_gemm_glu_f16", out, c["N"], t["a"], t["w"], t["w3"], c["M"], c["N"], c["K"], api.ACT_SILU if c["act"] == "silu" else api.ACT_GELU))
        s["out"] = out
    elif c["kind"] == "prompt_attention":
        out = torch.empty_like(t["q"])
        s["calls"].append(_call("yalm_attn_prefill", out, t["q"], t["k"], t["v"], c["n"], c["pos0"], c["heads"], c["kv_heads"], c["head_dim"], t["k"].shape[1]))
        s["out"] = out
    elif c["kind"] == "decode_attention":
        out = torch.empty_like(t["q"])
        bytes_ = api.lib().yalm_attn_workspace_bytes(c["heads"], c["kv_heads"], c["head_dim"])
        t["workspace"] = torch.zeros(bytes_, device="cuda", dtype=torch.uint8)
        t["ctl"] = torch.tensor([0, c["kv_len"] - 1, 0, c["kv_len"] - 1, c["kv_len"], 0, 0, 0], device="cuda", dtype=torch.int32)
        s["calls"].append(_call("yalm_attn_decode", out, t["k"], t["v"], t["q"], t["workspace"], c["heads"], c["kv_heads"], c["head_dim"], t["k"].shape[1], t["ctl"]))
        s["out"] = out
    elif c["kind"] == "window_attention":
        out = torch.empty((c["n"], c["heads"], c["dv"]), device="cuda")
        blocks = t["kp"].shape[1] if c["pool"] else 0
        s["calls"].append(_call("yalm_attn_window_pool_mma", out, c["heads"] * c["dv"], t["q"], c["heads"] * c["dk"], t["k"], t["v"], t.get("kp"), t.get("vp"),
                                c["n"], c["heads"], c["kv_heads"], c["dk"], c["dv"], t["k"].shape[1], blocks, c["window"], c["pool"], c["dk"] ** -0.5, c["pos0"], None))
        s["out"] = out
    elif c["kind"] == "scan":
        n, H, D, P = c["n"], c["heads"], c["D"], c["P"]
        out = torch.empty((n, H, P), device="cuda")
        per_channel = c["form"] != "delta_head"
        s["calls"].append(_call("yalm_state_scan_rows", out, H * P, t["k"], H * D, t["q"], H * D, t["v"], H * P, t["decay"], H * D if per_channel else H,
                                int(per_channel), None, 0, t.get("beta"), H if "beta" in t else 0, None, t["state"], n, H, 1, D, P, c["pos0"], None))
        s["out"] = [out, t["state"]]
    else:
        dim, hidden, code = c["dim"], c["hidden"], DTYPES[c["dtype"]][1]
        hb, out = torch.empty(hidden, device="cuda"), torch.empty(dim, device="cuda")
        s["calls"].append(_call("yalm_ffn_glu", hb, t["x"], t["norm"], t["w1"], t["w3"], t["s1"], t["s3"], None, None, dim, hidden,
                                api.ACT_SILU if c["act"] == "silu" else api.ACT_GELU, 1e-5, code, 0, 0, None, None, None))
        s["calls"].append(_call("yalm_gemv_residual", out, t["x"], hb, t["w2"], t["s2"], hidden, dim, code, 1, None, None))
        s["out"] = [out, hb]
    return s


def run(state):
    if "calls" in state:
        for fn, args in state["calls"]:
            rc = fn(*args)
            if rc:
                raise RuntimeError("%s: %d" % (fn.__name__, rc))
        return state["out"]
    s, ids = state["state"], state["ids"]
    if state["kind"] == "model_decode":
        return s.forward(int(ids[state["pos"]]), state["pos"]).copy()
    probs = s.forward_batch(ids, 0, state["targets"])
    return [s.logits().copy(), probs]


# ---- what a pass cannot do without ------------------------------------------------------------------------------------
def _visible(c):
    """(query, key) pairs of one head."""
    if c["kind"] == "window_attention":
        i = np.arange(c["pos0"], c["pos0"] + c["n"])
        pairs = np.minimum(i + 1, c["window"])
        if c["pool"]:
            pairs = pairs + np.maximum(0, i - c["window"] + 1) // c["pool"]
        return int(pairs.sum())
    return c["n"] * c["pos0"] + c["n"] * (c["n"] + 1) // 2


def work(case):
    c, kind = case, case["kind"]
    if kind == "gemm":
        M, N, K = c["M"], c["N"], c["K"]
        return {"bytes": 2 * (M * K + N * K) + 4 * M * N * (2 if c["accumulate"] else 1), "flops": 2 * M * N * K}
    if kind == "glu":
        M, N, K = c["M"], c["N"], c["K"]
        return {"bytes": 2 * (M * K + 2 * N * K + M * N), "flops": 4 * M * N * K}
    if kind == "prompt_attention":
        H, D = c["heads"], c["head_dim"]
        return {"bytes": 2 * (2 * c["n"] * H * D + 2 * (c["pos0"] + c["n"]) * c["kv_heads"] * D), "flops": 4 * _visible(c) * H * D}
    if kind == "decode_attention":
        H, D = c["heads"], c["head_dim"]
        return {"bytes": 2 * 2 * c["kv_len"] * c["kv_heads"] * D + 8 * H * D, "flops": 4 * c["kv_len"] * H * D}
    if kind == "window_attention":
        H, both = c["heads"], c["dk"] + c["dv"]
        first = max(0, c["pos0"] - c["window"] + 1)
        blocks = max(0, c["pos0"] + c["n"] - c["window"]) // c["pool"] if c["pool"] else 0
        return {"bytes": 4 * c["n"] * H * both + c["kv_heads"] * both * (2 * (c["pos0"] + c["n"] - first) + 4 * blocks), "flops": 2 * _visible(c) * H * both}
    if kind == "scan":
        n, H, D, P = c["n"], c["heads"], c["D"], c["P"]
        decay = 1 if c["form"] == "delta_head" else D
        return {"bytes": 4 * n * H * (2 * D + decay + 2 * P + 1) + 4 * H * D * P * (2 if c["pos0"] else 1),
                "flops": n * H * D * P * (5 if c["form"] == "linear_channel" else 7)}
    if kind == "decode_ffn":
        n = 3 * c["dim"] * c["hidden"]
        return {"bytes": n * DTYPES[c["dtype"]][2] + 4 * (4 * c["dim"] + c["hidden"]), "flops": 2 * n}
    q, kv = c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"]
    per_layer, head = c["dim"] * (2 * q + 2 * kv + 3 * c["hidden"]), c["vocab"] * c["dim"]
    if kind == "model_decode":
        rows = c["context"] + 1
        return {"bytes": 2 * (c["layers"] * (per_layer + 2 * rows * kv) + head + c["dim"]) + 4 * c["vocab"],
                "flops": 2 * (c["layers"] * (per_layer + 2 * rows * q) + head)}
    pairs = c["n"] * (c["n"] + 1) // 2
    return {"bytes": 2 * (c["layers"] * (per_layer + 4 * c["n"] * kv) + head + c["n"] * c["dim"]) + 4 * (c["vocab"] + 3 * c["n"]),
            "flops": 2 * c["n"] * (c["layers"] * per_layer + head) + 4 * c["layers"] * pairs * q}


def tolerance(case):
    # about four times the error measured against exact()
    kind = case["kind"]
    if kind in ("scan", "decode_attention", "decode_ffn"):
        return {"rel": 3e-6}  # 32-bit sums (4e-7)
    if kind == "gemm":
        return {"rel": 5e-5}  # the tensor cores' 32-bit sums, shortened at each addition (1.2e-5 at K = 14336)
    if kind in ("glu", "prompt_attention"):
        return {"rel": 1.2e-3}  # fp16 results (3e-4)
    if kind == "window_attention":
        return {"rel": 9e-3}  # bf16 queries and weights (2.2e-3)
    if kind == "model_decode":
        return {"rel": 3.5e-3}  # fp16 cached keys and values under it (9e-4)
    return {"rel": 6.5e-3}  # fp16 operands of every product (1.6e-3)


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------
def _act(x, act):
    # the library's tanh form with its rounded sqrt(2 / pi)
    return torch.nn.functional.silu(x) if act == "silu" else 0.5 * x * (1.0 + torch.tanh(0.797885 * (x + 0.044715 * x ** 3)))


def _attend(q, k, v, mask, scale):
    """q (n, H, dk), k (G, T, dk), v (G, T, dv), mask (n, T) or None -> (n, H, dv), head by head."""
    out = []
    rep = q.shape[1] // k.shape[0]
    for h in range(q.shape[1]):
        s = q[:, h] @ k[h // rep].T * scale
        if mask is not None:
            s = s.masked_fill(~mask, -math.inf)
        out.append(torch.softmax(s, dim=-1) @ v[h // rep])
    return torch.stack(out, dim=1)


def _rms(x, w):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + 1e-5) * w


def _rope(x, theta):
    """x (n, heads, size), rows at positions 0 .. n - 1, neighbouring pairs turned."""
    n, _, size = x.shape
    angle = torch.arange(n, device=x.device, dtype=torch.float64)[:, None] * theta ** (-torch.arange(0, size, 2, device=x.device, dtype=torch.float64) / size)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack([a * cos - b * sin, a * sin + b * cos], dim=-1).reshape(x.shape)


def _exact_model(c, seed):
    W = dict(_model_tensors(c, seed))
    ids, targets = _tokens(c, seed)
    n, H, G, D = len(ids), c["heads"], c["kv_heads"], c["head_dim"]
    x = W["model.embed.weight"][torch.from_numpy(ids).long().cuda()].double()
    mask = torch.ones((n, n), dtype=torch.bool, device="cuda").tril()
    for l in range(c["layers"]):
        w = lambda name: W["model.layers.%d.%s.weight" % (l, name)].double()  # noqa: B023,E731
        y = _rms(x, w("attn.norm"))
        q, k, v = _rope((y @ w("attn.wq").T).view(n, H, D), 1e6), _rope((y @ w("attn.wk").T).view(n, G, D), 1e6), (y @ w("attn.wv").T).view(n, G, D)
        x = x + _attend(q, k.transpose(0, 1), v.transpose(0, 1), mask, D ** -0.5).reshape(n, H * D) @ w("attn.wo").T
        y = _rms(x, w("mlp.norm"))
        x = x + (_act(y @ w("mlp.w1").T, "silu") * (y @ w("mlp.w3").T)) @ w("mlp.w2").T
    y = _rms(x, W["model.norm.weight"].double())
    if c["kind"] == "model_decode":
        return y[-1] @ W["model.output.weight"].double().T
    logits = y @ W["model.output.weight"].double().T
    probs = torch.softmax(logits, dim=-1).gather(1, torch.from_numpy(targets).long().cuda()[:, None])[:, 0]
    return [logits[-1], probs]


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("model_decode", "model_prompt"):
        return _exact_model(c, seed)
    t = _inputs(c, seed)
    if kind == "gemm":
        return t["c"].double() + t["a"].double() @ t["w"].double().T
    if kind == "glu":
        a = t["a"].double()
        return _act(a @ t["w"].double().T, c["act"]) * (a @ t["w3"].double().T)
    if kind == "prompt_attention":
        rows, i = c["pos0"] + c["n"], torch.arange(c["n"], device="cuda")
        mask = torch.arange(rows, device="cuda")[None] <= (c["pos0"] + i)[:, None]
        return _attend(t["q"].double(), t["k"][:, :rows].double(), t["v"][:, :rows].double(), mask, c["head_dim"] ** -0.5)
    if kind == "decode_attention":
        return _attend(t["q"].double(), t["k"][:, : c["kv_len"]].double(), t["v"][:, : c["kv_len"]].double(), None, c["head_dim"] ** -0.5)
    if kind == "window_attention":
        pos = torch.arange(c["pos0"], c["pos0"] + c["n"], device="cuda")[:, None]
        first = max(0, c["pos0"] - c["window"] + 1)
        j = torch.arange(first, c["pos0"] + c["n"], device="cuda")
        slot = j % t["k"].shape[1]
        k, v, mask = t["k"][:, slot].double(), t["v"][:, slot].double(), (j[None] <= pos) & (pos - j[None] < c["window"])
        if c["pool"]:
            b = torch.arange(t["kp"].shape[1], device="cuda")[None]
            k, v = torch.cat([k, t["kp"].double()], dim=1), torch.cat([v, t["vp"].double()], dim=1)
            mask = torch.cat([mask, b * c["pool"] + c["pool"] - 1 <= pos - c["window"]], dim=1)
        return _attend(t["q"].double(), k, v, mask, c["dk"] ** -0.5)
    if kind == "scan":
        k, q, v, decay = (t[x].double() for x in ("k", "q", "v", "decay"))
        S = t["state"].double() if c["pos0"] else torch.zeros_like(t["state"], dtype=torch.float64)  # (head, column, row)
        out = []
        for i in range(c["n"]):
            S = S * (decay[i][:, None, :] if decay.dim() == 3 else decay[i][:, None, None])
            e = v[i]
            if "beta" in t:
                e = t["beta"][i].double()[:, None] * (e - torch.einsum("hpd,hd->hp", S, k[i]))
            S = S + e[:, :, None] * k[i][:, None, :]
            out.append(torch.einsum("hpd,hd->hp", S, q[i]))
        return [torch.stack(out), S]
    x = t["x"].double()
    y = _rms(x, t["norm"].double())
    hb = _act(_plain(t["w1"], t["s1"]) @ y, c["act"]) * (_plain(t["w3"], t["s3"]) @ y)
    return [x + _plain(t["w2"], t["s2"]) @ hb, hb]
