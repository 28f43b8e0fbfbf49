"""Workloads of the grouped dual-NVFP4 GEMM library, as a serving or training program calls it.

Five kinds, one per public entry point:

  gemm      m_grouped_bf16_dual_nvfp4_gemm_contiguous, normal orientation (prefill)
  decode    the same call with tune_swap_ab=1 (a few tokens per expert)
  masked    m_grouped_bf16_dual_nvfp4_gemm_masked (fixed rows per expert, row counts on the device)
  layer     ep.ExpertParallelMoE, the whole expert layer: dispatch, up, SwiGLU, down, combine
  quantize  quantize_weight_nvfp4 (loading a model's BF16 / FP32 expert weights)

``listed()`` gives fixed sizes, ``draw(rng)`` others out of the same ranges.  Routing, activations and weights
come from the seed; weights are what a program quantises once when it loads its model, so they belong to
``prepare`` (except where quantising them is the workload).
"""
import math

import torch

import nvfp4_gemm
from nvfp4_cutlass_b200.ep import ExpertParallelMoE

WEIGHT_STD = 0.02
CHUNK = 1 << 28            # weight elements made at a time


def listed():
    return [
        # one decode step of a small batch, gate+up of a 256-expert model with 32 experts on this GPU: the smallest call
        {"name": "decode_16_tokens", "kind": "decode", "experts": 32, "experts_total": 256, "top_k": 8, "tokens": 16,
         "n": 1024, "k": 2048, "align": 16, "residual": True},
        # the down projection of the same model at a larger batch, with the entry point's default row alignment
        {"name": "decode_128_tokens_down", "kind": "decode", "experts": 32, "experts_total": 256, "top_k": 8,
         "tokens": 128, "n": 2048, "k": 512, "align": 32, "residual": True},
        # decode of a DeepSeek-V3-sized layer with all 256 experts on one GPU: streams 3.6 GB of weights
        {"name": "decode_64_tokens_256_experts", "kind": "decode", "experts": 256, "experts_total": 256, "top_k": 8,
         "tokens": 64, "n": 4096, "k": 7168, "align": 16, "residual": True},
        # prefill of the small-expert model, balanced rows (the reference's own sweep): gate+up
        {"name": "prefill_8k_rows_up", "kind": "gemm", "experts": 32, "rows": 8192, "routing": "balanced", "n": 1024,
         "k": 2048, "align": 128, "policy": "derived_div8", "residual": True},
        # its down projection with the rows a router really gives: ragged groups padded to 128
        {"name": "prefill_16k_rows_down", "kind": "gemm", "experts": 32, "rows": 16384, "routing": "uniform", "n": 2048,
         "k": 512, "align": 128, "policy": "derived_div8", "residual": True},
        # Mixtral-8x7B-like gate+up: eight wide experts, the tensor-bound prefill
        {"name": "prefill_4k_rows_wide", "kind": "gemm", "experts": 8, "rows": 4096, "routing": "balanced", "n": 28672,
         "k": 4096, "align": 256, "policy": "derived_div8", "residual": True},
        # DeepSeek-V3-like prefill, 4096 tokens over 256 experts with a skewed router: gate+up
        {"name": "prefill_32k_rows_zipf_up", "kind": "gemm", "experts": 256, "rows": 32768, "routing": "zipf", "n": 4096,
         "k": 7168, "align": 128, "policy": "derived_div8", "residual": True},
        # its down projection with the residual pass off (the single_nvfp4 mode)
        {"name": "prefill_32k_rows_zipf_down_single", "kind": "gemm", "experts": 256, "rows": 32768, "routing": "zipf",
         "n": 7168, "k": 2048, "align": 128, "policy": "derived_div8", "residual": False},
        # masked layout: an engine that captured its step in a graph hands over row counts on the device
        {"name": "masked_32_groups", "kind": "masked", "experts": 32, "max_m": 1024, "rows": 16384, "n": 3072, "k": 4096,
         "residual": True},
        # Qwen3-235B-like expert layer, prefill: the largest workload
        {"name": "layer_16k_tokens", "kind": "layer", "experts": 128, "hidden": 4096, "inter": 1536, "tokens": 16384,
         "top_k": 8},
        # the same layer while decoding a batch of 256 sequences
        {"name": "layer_256_tokens", "kind": "layer", "experts": 128, "hidden": 4096, "inter": 1536, "tokens": 256,
         "top_k": 8},
        # loading a model: the gate+up weights of eight experts
        {"name": "quantize_8_experts", "kind": "quantize", "experts": 8, "n": 4096, "k": 7168, "dtype": "bfloat16"},
    ]


def _log_int(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi // step * step, max(-(-lo // step) * step, int(v / step + 0.5) * step))


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["gemm", "gemm", "gemm", "decode", "decode", "masked", "layer", "layer", "quantize"])
        if kind == "gemm":
            c = {"kind": kind, "experts": _log_int(rng, 4, 256), "rows": _log_int(rng, 512, 32768),
                 "routing": rng.choice(["balanced", "uniform", "zipf"]), "n": _log_int(rng, 512, 28672, 128),
                 "k": _log_int(rng, 512, 7168, 128), "align": 128,
                 "policy": rng.choice(["derived_div8"] * 5 + ["residual_amax"]), "residual": rng.random() < 0.75}
        elif kind == "decode":
            total = _log_int(rng, 32, 256, 8)
            c = {"kind": kind, "experts": total // rng.choice([1, 2, 8]), "experts_total": total,
                 "top_k": rng.choice([4, 8]), "tokens": _log_int(rng, 4, 128), "n": _log_int(rng, 512, 7168, 128),
                 "k": _log_int(rng, 512, 7168, 128), "align": rng.choice([16, 32]), "residual": rng.random() < 0.75}
        elif kind == "masked":
            experts, max_m = _log_int(rng, 8, 128), _log_int(rng, 128, 2048, 128)
            c = {"kind": kind, "experts": experts, "max_m": max_m,
                 "rows": _log_int(rng, max(experts, experts * max_m // 16), experts * max_m * 3 // 4),
                 "n": _log_int(rng, 512, 7168, 256), "k": _log_int(rng, 512, 7168, 128), "residual": rng.random() < 0.75}
        elif kind == "layer":
            c = {"kind": kind, "experts": _log_int(rng, 16, 128, 8), "hidden": 1024 * rng.randint(1, 4),
                 "inter": _log_int(rng, 512, 2048, 128), "tokens": _log_int(rng, 32, 16384), "top_k": rng.choice([4, 8])}
        else:
            c = {"kind": kind, "experts": _log_int(rng, 1, 16), "n": _log_int(rng, 512, 8192, 64),
                 "k": _log_int(rng, 512, 7168, 64), "dtype": rng.choice(["bfloat16", "bfloat16", "float32"])}
        if _cost(c) <= most and _weight_elements(c) <= 256 * 4096 * 7168:
            return c


def _weight_elements(c):
    if c["kind"] == "layer":
        return c["experts"] * 3 * c["hidden"] * c["inter"]
    return c["experts"] * c["n"] * c["k"]


def _cost(c):
    w = work(c)
    return max(w["bytes"], w["flops"] / 50)


# ------------------------------------------------------------------------------------------------- inputs
def _weights(experts, n, k, gen, dtype=torch.bfloat16):
    """Quantised weights (b, sfb, gw) of `experts` (n, k) matrices ~ N(0, 0.02), made a few experts at a time."""
    step = max(1, CHUNK // (n * k))
    parts = []
    for e in range(0, experts, step):
        w = torch.randn(min(step, experts - e), n, k, generator=gen, device="cuda", dtype=dtype).mul_(WEIGHT_STD)
        parts.append(nvfp4_gemm.quantize_weight_nvfp4(w))
    return tuple(torch.cat(t) for t in zip(*parts))


def _activations(rows, k, gen):
    """BF16 rows ~ N(0, 1) with a lognormal scale per row and one channel in a thousand 50 times as large."""
    x = torch.randn(rows, k, generator=gen, device="cuda", dtype=torch.bfloat16)
    x *= torch.exp(0.5 * torch.randn(rows, 1, generator=gen, device="cuda")).to(torch.bfloat16)
    x[:, torch.randperm(k, generator=gen, device="cuda")[:max(1, k // 1000)]] *= 50.0
    return x.clamp_(-2688.0, 2688.0)


def _group_sizes(c, seed):
    """Real rows per expert.  The multiset of sizes belongs to the case, so that the output keeps its shape; which expert
    gets which size comes from the seed."""
    e, gen = c["experts"], torch.Generator().manual_seed(c.get("rows", c.get("tokens")))
    if c["kind"] == "decode":                    # every token picks top_k different experts of all; `experts` live here
        picks = torch.rand(c["tokens"], c["experts_total"], generator=gen).topk(c["top_k"], dim=1).indices
        sizes = picks.flatten().bincount(minlength=c["experts_total"])[:e]
        if int(sizes.sum()) == 0:                # all tokens went to other GPUs: keep one row
            sizes[0] = 1
    elif c.get("routing") == "balanced":
        sizes = torch.full((e,), c["rows"] // e) + (torch.arange(e) < c["rows"] % e)
    else:
        p = torch.arange(1, e + 1, dtype=torch.float64).pow(-1.1 if c.get("routing") == "zipf" else 0.0)
        sizes = torch.multinomial(p / p.sum(), c["rows"], replacement=True, generator=gen).bincount(minlength=e)
    return sizes[torch.randperm(e, generator=torch.Generator().manual_seed(seed))]


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if c["kind"] == "quantize":
        return {"case": c, "w": torch.randn(c["experts"], c["n"], c["k"], generator=gen, device="cuda",
                                            dtype=getattr(torch, c["dtype"])).mul_(WEIGHT_STD)}
    if c["kind"] == "layer":
        return _prepare_layer(c, gen)
    b, sfb, gw = _weights(c["experts"], c["n"], c["k"], gen)
    real = _group_sizes(c, seed)
    state = {"case": c, "b": b, "sfb": sfb, "gw": gw}
    if c["kind"] == "masked":
        real = real.clamp(max=c["max_m"])
        rows = c["experts"] * c["max_m"]
        place = torch.cat([torch.arange(r) + g * c["max_m"] for g, r in enumerate(real.tolist())])
        shape = (c["experts"], c["max_m"])
        state["masked_m"] = real.to(torch.int32).cuda()
    else:
        padded = (real + c["align"] - 1) // c["align"] * c["align"]
        rows = int(padded.sum())
        start = padded.cumsum(0) - padded
        place = torch.cat([torch.arange(r) + s for r, s in zip(real.tolist(), start.tolist())])
        shape = (rows,)
        state["m_indices"] = nvfp4_gemm.make_m_indices(padded, device="cuda", alignment=c["align"])
    a = torch.zeros(rows, c["k"], dtype=torch.bfloat16, device="cuda")
    a[place.cuda()] = _activations(place.numel(), c["k"], gen)
    state["a"] = a.view(*shape, c["k"])
    state["d"] = torch.zeros(*shape, c["n"], dtype=torch.bfloat16, device="cuda")
    return state


def _prepare_layer(c, gen):
    up = _weights(c["experts"], 2 * c["inter"], c["hidden"], gen)
    down = _weights(c["experts"], c["hidden"], c["inter"], gen)
    average = c["tokens"] * c["top_k"] // c["experts"]
    layer = ExpertParallelMoE(c["experts"], c["hidden"], c["inter"], up, down, peer_rows_cap=average * 3 // 2 + 128)
    x = _activations(c["tokens"], c["hidden"], gen)
    scores = torch.softmax(torch.randn(c["tokens"], c["experts"], generator=gen, device="cuda"), dim=-1)
    w, ids = torch.topk(scores, c["top_k"], dim=-1)
    return {"case": c, "layer": layer, "x": x, "ids": ids, "w": w / w.sum(dim=-1, keepdim=True)}


# ------------------------------------------------------------------------------------------------- one pass
def run(state):
    c = state["case"]
    if c["kind"] == "quantize":
        return nvfp4_gemm.quantize_weight_nvfp4(state["w"])
    if c["kind"] == "layer":
        return state["layer"](state["x"], state["ids"], state["w"])
    a, b, sfb, gw, d = (state[name] for name in ("a", "b", "sfb", "gw", "d"))
    if c["kind"] == "masked":
        nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_masked(a, b, sfb, gw, d, state["masked_m"],
                                                         enable_residual_pass=c["residual"])
    elif c["kind"] == "decode":
        nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(a, b, sfb, gw, d, state["m_indices"],
                                                             enable_residual_pass=c["residual"],
                                                             m_alignment=c["align"], tune_swap_ab=1)
    else:
        nvfp4_gemm.m_grouped_bf16_dual_nvfp4_gemm_contiguous(a, b, sfb, gw, d, state["m_indices"], c["policy"],
                                                             c["residual"], m_alignment=c["align"])
    return d


# ------------------------------------------------------------------------------------------------- accounting
def work(case):
    """Bytes: weights of the experts that get rows (4 bits a code, one scale byte per 16), real activation rows in and
    out.  Operations: one multiply-add per real row, weight and NVFP4 pass.  Routing enters by its expectation."""
    c = case
    if c["kind"] == "quantize":
        elements = c["experts"] * c["n"] * c["k"]
        return {"bytes": elements * ((2 if c["dtype"] == "bfloat16" else 4) + 9 / 16), "flops": 4 * elements}
    if c["kind"] == "layer":
        pairs = c["tokens"] * c["top_k"]
        elements = 3 * c["hidden"] * c["inter"]
        active = c["experts"] * (1 - (1 - c["top_k"] / c["experts"]) ** c["tokens"])
        return {"bytes": active * elements * 9 / 16 + 4 * c["tokens"] * c["hidden"] + 12 * pairs, "flops": 4 * pairs * elements}
    if c["kind"] == "decode":
        rows = c["tokens"] * c["top_k"] * c["experts"] / c["experts_total"]
        active = c["experts"] * (1 - (1 - c["top_k"] / c["experts_total"]) ** c["tokens"])
    else:
        rows, e = c["rows"], c["experts"]
        p = [r ** -1.1 if c.get("routing") == "zipf" else 1.0 for r in range(1, e + 1)]
        active = e if c.get("routing") == "balanced" else sum(1 - (1 - q / sum(p)) ** rows for q in p)
    return {"bytes": active * c["n"] * c["k"] * 9 / 16 + 2 * rows * (c["k"] + c["n"]),
            "flops": 2 * rows * c["n"] * c["k"] * (2 if c["residual"] else 1)}


def tolerance(case):
    if case["kind"] == "quantize":
        return "exact"                           # codes, scales and global scales are defined bit for bit
    if case["kind"] == "layer":                  # a BF16 tie between the projections can move a four-bit code
        return {"rel": 1e-2, "max": 0.1}
    # exact four-bit products summed in FP32 in any order, then one rounding to BF16 (half an ulp either way)
    return {"rel": 3e-3, "max": 0.02}
