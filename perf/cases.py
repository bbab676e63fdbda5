"""The work that a user of this framework gives it, as cases that can be timed and compared.

A case is a dict of plain values; ``kind`` says which path of an FP8 inference server it stands for:

  block_linear    a linear layer of a block-FP8 model (DeepSeek-V3): 16-bit activations are quantised per 1x128
                  group, then multiplied by a weight with 128x128 block scales
  channel_linear  a linear layer of a per-channel FP8 model (Llama-3-8B): activations quantised per token
                  (``scales`` = "token") or with the checkpoint's one static scale ("tensor"), then the scaled product
  quant           activation quantisation alone, as a model calls it in front of a kernel of its own
  moe             the MoE block of a server: router, then ``fused_experts_impl``
  layer           the same block through ``ExpertParallelMoE`` on one GPU, with its shared expert
  grouped_mm      aten ``_scaled_grouped_mm``: rows sorted by group against one weight per group

Inputs are synthetic with the distributions that the path meets: activations N(0, 1), weights N(0, 0.02)
quantised to e4m3, router logits with the skew of the model that the case stands for.
"""
import math
import random

import numpy as np
import torch

import flag_gems
from flaggems_b200.ep import ExpertParallelMoE

FP8 = torch.float8_e4m3fn
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
# (outputs, inputs) of the linear layers: DeepSeek-V3 projections, a DeepSeek-V3 shared expert, Llama-3-8B
BLOCK_SHAPES = ((2112, 7168), (4096, 7168), (18432, 7168), (24576, 7168), (7168, 2048))
CHANNEL_SHAPES = ((6144, 4096), (4096, 4096), (28672, 4096), (4096, 14336))
# expert layers: hidden size, intermediate size, experts, experts per token
DEEPSEEK = {"hidden": 7168, "inter": 2048, "experts": 256, "topk": 8}
MIXTRAL = {"hidden": 4096, "inter": 14336, "experts": 8, "topk": 2}


def listed():
    return [
        # One token through the smallest projection: launches and the host path are most of it.
        {"name": "block_linear_1x2112", "kind": "block_linear", "m": 1, "n": 2112, "k": 7168, "dtype": "bf16"},
        # A decode batch through the widest projection: the weight has to be streamed.
        {"name": "block_linear_64x24576", "kind": "block_linear", "m": 64, "n": 24576, "k": 7168, "dtype": "bf16"},
        # A prefill chunk through a wide projection: tensor cores.
        {"name": "block_linear_4096x18432", "kind": "block_linear", "m": 4096, "n": 18432, "k": 7168, "dtype": "bf16"},
        # A decode batch of a dense model, gate_up projection.
        {"name": "channel_linear_16x28672", "kind": "channel_linear", "m": 16, "n": 28672, "k": 4096,
         "dtype": "bf16", "scales": "token", "bias": False},
        # A short prompt of odd length, qkv projection with bias.
        {"name": "channel_linear_1037x6144", "kind": "channel_linear", "m": 1037, "n": 6144, "k": 4096,
         "dtype": "bf16", "scales": "token", "bias": True},
        # A full prefill batch, down projection.
        {"name": "channel_linear_8192x4096", "kind": "channel_linear", "m": 8192, "n": 4096, "k": 14336,
         "dtype": "bf16", "scales": "token", "bias": False},
        # The activations of a prefill batch quantised on their own.
        {"name": "act_quant_16384x7168", "kind": "quant", "m": 16384, "k": 7168, "dtype": "bf16", "form": "act"},
        # A decode batch of DeepSeek-V3: a few rows for each of many experts.
        {"name": "deepseek_moe_32", "kind": "moe", "tokens": 32, "mode": "block", "dtype": "bf16", **DEEPSEEK},
        # A decode batch of odd size with unquantised experts.
        {"name": "mixtral_moe_bf16_129", "kind": "moe", "tokens": 129, "mode": "plain", "dtype": "bf16", **MIXTRAL},
        # Prefill of Mixtral-8x7B, per-token x per-channel FP8.
        {"name": "mixtral_moe_fp8_4096", "kind": "moe", "tokens": 4096, "mode": "channel", "dtype": "bf16", **MIXTRAL},
        # Prefill of DeepSeek-V3, the layer with its shared expert: the largest.
        {"name": "deepseek_layer_8192", "kind": "layer", "tokens": 8192, "mode": "block", "dtype": "bf16", **DEEPSEEK},
        # Grouped product over ragged groups, as a framework that sorts its own tokens calls it.
        {"name": "grouped_mm_8192", "kind": "grouped_mm", "m": 8192, "n": 4096, "k": 7168, "groups": 32},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    kind = rng.choice(("block_linear", "block_linear", "block_linear", "channel_linear", "channel_linear",
                       "channel_linear", "quant", "moe", "moe", "moe", "moe", "layer", "grouped_mm"))
    dtype = rng.choice(("bf16", "bf16", "bf16", "fp16"))
    if kind == "block_linear":
        n, k = rng.choice(BLOCK_SHAPES)
        return {"kind": kind, "m": _log_int(rng, 1, 16384), "n": n, "k": k, "dtype": dtype}
    if kind == "channel_linear":
        n, k = rng.choice(CHANNEL_SHAPES)
        return {"kind": kind, "m": _log_int(rng, 1, 8192), "n": n, "k": k, "dtype": dtype,
                "scales": rng.choice(("token", "token", "tensor")), "bias": rng.random() < 0.3}
    if kind == "quant":
        return {"kind": kind, "m": _log_int(rng, 1, 16384), "k": rng.choice((2048, 4096, 7168, 14336)),
                "dtype": "bf16", "form": rng.choice(("act", "act", "group", "group_ue8m0", "group_column"))}
    if kind == "moe":
        if rng.random() < 0.5:
            return {"kind": kind, "tokens": _log_int(rng, 1, 8192), "mode": "block", "dtype": dtype, **DEEPSEEK}
        return {"kind": kind, "tokens": _log_int(rng, 1, 4096),
                "mode": rng.choice(("channel", "channel", "int8", "plain", "tensor")), "dtype": dtype, **MIXTRAL}
    if kind == "layer":
        return {"kind": kind, "tokens": _log_int(rng, 1, 8191), "mode": "block", "dtype": "bf16", **DEEPSEEK}
    return {"kind": kind, "m": _log_int(rng, 64, 16384), "n": rng.choice((2048, 4096)),
            "k": rng.choice((2048, 4096, 7168)), "groups": rng.choice((8, 16, 32))}


# ---- inputs ---------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _randn(g, *shape, scale=1.0):
    return torch.randn(*shape, device="cuda", generator=g) * scale


def _quantize_block(w):
    """[N, K] -> e4m3 [N, K] and fp32 [ceil(N / 128), K / 128] (one scale per 128x128 block)."""
    n, k = w.shape
    rows = (n + 127) // 128 * 128
    t = torch.nn.functional.pad(w, (0, 0, 0, rows - n)).view(rows // 128, 128, k // 128, 128)
    s = t.abs().amax(dim=(1, 3)).clamp_min(1e-10) / 448.0
    return (t / s[:, None, :, None]).view(rows, k)[:n].to(FP8), s


def _quantize_channel(w, top=448.0, dtype=FP8):
    s = w.abs().amax(1).clamp_min(1e-10) / top
    q = w / s[:, None]
    return (q.round() if dtype == torch.int8 else q).to(dtype), s


def _block_weight(g, n, k):
    return _quantize_block(_randn(g, n, k, scale=0.02))


def _experts(g, case):
    """The expert weights of a case and the arguments that say how they are stored."""
    e, h, i, mode = case["experts"], case["hidden"], case["inter"], case["mode"]
    stored = {"block": FP8, "channel": FP8, "tensor": FP8, "int8": torch.int8, "plain": DTYPES[case["dtype"]]}[mode]
    w1 = torch.empty(e, 2 * i, h, dtype=stored, device="cuda")
    w2 = torch.empty(e, h, i, dtype=stored, device="cuda")
    scales = ([], [])
    for x in range(e):
        for w, s in ((w1, scales[0]), (w2, scales[1])):
            v = _randn(g, *w.shape[1:], scale=0.02)
            if mode == "block":
                w[x], sx = _quantize_block(v)
            elif mode == "channel":
                w[x], sx = _quantize_channel(v)
            elif mode == "int8":
                w[x], sx = _quantize_channel(v, 127.0, torch.int8)
            elif mode == "tensor":
                sx = v.abs().max() / 448.0
                w[x] = (v / sx).to(FP8)
            else:
                w[x], sx = v.to(stored), None
            s.append(sx)
    if mode == "plain":
        return w1, w2, {}
    how = {"w1_scale": torch.stack(scales[0]), "w2_scale": torch.stack(scales[1])}
    if mode == "int8":
        how.update(use_int8_w8a8=True, per_channel_quant=True)
    else:
        how.update(use_fp8_w8a8=True, per_channel_quant=mode == "channel")
    if mode == "block":
        how["block_shape"] = [128, 128]
    return w1, w2, how


def _popularity(experts):
    """Zipf(1.1) popularity of the experts in a fixed shuffled order (a large router is skewed)."""
    p = np.arange(1, experts + 1, dtype=np.float64) ** -1.1
    return np.random.RandomState(0).permutation(p / p.sum())


def _router_inputs(g, case):
    """Router logits: Gumbel noise on a Zipf popularity for the many-expert model, N(0, 1) for the small one."""
    t, e = case["tokens"], case["experts"]
    if e <= 32:
        return {"logits": _randn(g, t, e)}
    u = torch.rand(t, e, device="cuda", generator=g).clamp_min(1e-9)
    logp = torch.from_numpy(np.log(_popularity(e)) + math.log(e)).float().cuda()
    return {"logits": logp - torch.log(-torch.log(u)), "bias": _randn(g, e, scale=0.01)}


def _route(case, s):
    """Router weights and expert ids of a step: group-limited sigmoid top-k (DeepSeek-V3) or softmax top-k."""
    if "bias" in s:
        return flag_gems.grouped_topk(s["logits"], 8, 4, case["topk"], True, 2.5, s["bias"], 1)
    t, k = case["tokens"], case["topk"]
    weights = torch.empty(t, k, device="cuda")
    ids = torch.empty(t, k, dtype=torch.int32, device="cuda")
    source = torch.empty(t, k, dtype=torch.int32, device="cuda")
    flag_gems.topk_softmax(weights, ids, source, s["logits"], True)
    return weights, ids


def prepare(case, seed):
    g, kind = _generator(seed), case["kind"]
    s = {"case": case}
    if kind == "block_linear":
        s["x"] = _randn(g, case["m"], case["k"]).to(DTYPES[case["dtype"]])
        s["w"], s["ws"] = _block_weight(g, case["n"], case["k"])
    elif kind == "channel_linear":
        dtype = DTYPES[case["dtype"]]
        s["x"] = _randn(g, case["m"], case["k"]).to(dtype)
        w = _randn(g, case["n"], case["k"], scale=0.02)
        if case["scales"] == "token":
            w, s["ws"] = _quantize_channel(w)
        else:
            s["ws"] = (w.abs().max() / 448.0).reshape(1)
            w = (w / s["ws"]).to(FP8)
            s["xs"] = torch.full((1,), 6.0 / 448.0, device="cuda")  # calibrated: activations beyond +-6 are rare
        s["wt"] = w.t()
        s["bias"] = _randn(g, case["n"]).to(dtype) if case["bias"] else None
    elif kind == "quant":
        s["x"] = _randn(g, case["m"], case["k"]).to(DTYPES[case["dtype"]])
    elif kind in ("moe", "layer"):
        s["x"] = _randn(g, case["tokens"], case["hidden"]).to(DTYPES[case["dtype"]])
        s.update(_router_inputs(g, case))
        w1, w2, how = _experts(g, case)
        if kind == "moe":
            s["w1"], s["w2"], s["how"] = w1, w2, how
        else:
            a, sa = _block_weight(g, 2 * case["inter"], case["hidden"])
            b, sb = _block_weight(g, case["hidden"], case["inter"])
            s["layer"] = ExpertParallelMoE(w1, w2, how["w1_scale"], how["w2_scale"], case["experts"],
                                           shared=(a, b, sa, sb))
    else:
        m, n, k, groups = case["m"], case["n"], case["k"], case["groups"]
        x = _randn(g, m, k)
        xs = x.abs().amax(1).clamp_min(1e-10) / 448.0
        s["a"], s["sa"] = (x / xs[:, None]).to(FP8), xs
        b = torch.empty(groups, n, k, dtype=FP8, device="cuda")
        sb = torch.empty(groups, n, device="cuda")
        for i in range(groups):
            b[i], sb[i] = _quantize_channel(_randn(g, n, k, scale=0.02))
        s["b"], s["sb"] = b.transpose(1, 2), sb
        cuts = torch.randint(0, m + 1, (groups - 1,), device="cuda", generator=g).sort().values
        s["offs"] = torch.cat([cuts, cuts.new_full((1,), m)]).to(torch.int32)
    return s


# ---- one pass -------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "block_linear":
        q, qs = flag_gems.per_token_group_quant_fp8(s["x"], 128)
        return flag_gems.w8a8_block_fp8_matmul(q, s["w"], qs, s["ws"], [128, 128], s["x"].dtype)
    if kind == "channel_linear":
        x = s["x"]
        if case["scales"] == "tensor":
            q, qs = flag_gems.moe_kernel_quantize_input(x, s["xs"], FP8, False)
            return flag_gems.scaled_mm(q, s["wt"], qs, s["ws"], s["bias"], None, x.dtype)
        q, qs = flag_gems.moe_kernel_quantize_input(x, None, FP8, True)
        out = torch.empty(case["m"], case["n"], dtype=x.dtype, device=x.device)
        flag_gems.cutlass_scaled_mm(out, q, s["wt"], qs, s["ws"], s["bias"])
        return out
    if kind == "quant":
        if case["form"] == "act":
            return flag_gems.act_quant_triton(s["x"], 128)
        return flag_gems.per_token_group_quant_fp8(s["x"], 128, column_major_scales=case["form"] == "group_column",
                                                   scale_ue8m0=case["form"] == "group_ue8m0")
    if kind == "moe":
        weights, ids = _route(case, s)
        return flag_gems.fused_experts_impl(s["x"], s["w1"], s["w2"], weights, ids, **s["how"])
    if kind == "layer":
        weights, ids = _route(case, s)
        return s["layer"](s["x"], weights, ids)
    return flag_gems.scaled_grouped_mm(s["a"], s["b"], s["sa"], s["sb"], s["offs"], out_dtype=torch.bfloat16)


# ---- what a pass cannot do without ----------------------------------------------------------
def _experts_hit(case):
    """Experts that a step of this size routes at least one token to, on average."""
    t, e, k = case["tokens"], case["experts"], case["topk"]
    if e <= 32:
        return e * (1.0 - (1.0 - k / e) ** t)
    r = np.random.RandomState(1)
    hits = []
    for _ in range(4):
        score = np.log(_popularity(e)) + r.gumbel(size=(min(t, 2048), e))
        group = np.sort(score.reshape(len(score), 8, -1), axis=2)[:, :, -2:].sum(2)
        score[np.repeat(group < np.sort(group, axis=1)[:, 4:5], e // 8, axis=1)] = -np.inf
        hits.append(len(np.unique(np.argpartition(-score, k, axis=1)[:, :k])))
    return float(np.mean(hits))


def work(case):
    kind = case["kind"]
    if kind in ("block_linear", "channel_linear"):
        m, n, k = case["m"], case["n"], case["k"]
        scales = n * k / 128 / 128 if kind == "block_linear" else n
        return {"bytes": 2 * m * k + n * k + 4 * scales + 2 * m * n, "flops": 2 * m * n * k}
    if kind == "quant":
        return {"bytes": case["m"] * case["k"] * (3 + 4 / 128), "flops": 0}
    if kind in ("moe", "layer"):
        t, h, i, k = case["tokens"], case["hidden"], case["inter"], case["topk"]
        size = 2 if case["mode"] == "plain" else 1
        experts, rows = _experts_hit(case), t * k
        if kind == "layer":
            experts, rows = experts + 1, rows + t
        return {"bytes": experts * 3 * h * i * size + 4 * t * h + 4 * t * case["experts"], "flops": 6 * rows * h * i}
    m, n, k, groups = case["m"], case["n"], case["k"], case["groups"]
    used = min(groups, m)
    return {"bytes": m * k + used * n * k + 4 * (m + used * n) + 2 * m * n, "flops": 2 * m * n * k}


def tolerance(case):
    # Quantised bytes and scales are defined bit for bit; products end in a 16-bit rounding.
    return "exact" if case["kind"] == "quant" else {"rel": 1e-2}
