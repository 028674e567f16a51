"""Performance cases of the fused MoE FFN layer, through the public Python entry points.

Three ways the layer is used:

  bf16    inference, bf16 weights: router logits -> ``route_topk_align`` -> ``fused_moe_bf16``
  mxfp8   inference, OCP-MX weights: the same with ``quantize_mx`` of the bf16 activations and ``fused_moe_mxfp8``
  train   bf16 forward and backward through the autograd layer ``moe_ffn`` (gradients of x, both weights and the
          routing weights); the gate/up pre-activations are kept for the backward pass on narrow layers with full
          experts and recomputed where keeping them is dear: wide layers, and experts that are mostly padding

A case is a layer (K hidden size, E experts, N = gate + up rows of one expert, top_k), a number of tokens T and a
routing distribution. The layers are the ones ``bench.py`` names; ``draw`` spreads all sizes over the range those span.
Weights, activations and logits are seeded Gaussians of the scale the layers meet (w ~ N(0, 1/fan_in), x ~ N(0, 1));
"zipf" routing prefers expert e with weight (e+1)^-1.2, sampled without replacement per token.
"""
import math

import torch

import prime_flash_moe_b200 as P

#        K     E    N      top_k
C0 = (4096, 8, 512, 4)           # a few narrow experts, launch-bound
C1 = (4096, 8, 28672, 2)         # few wide experts
C2 = (2048, 128, 1536, 8)        # many narrow experts
C3 = (7168, 256, 4096, 8)        # many experts of ordinary width, mxfp8 weights (11 GB)
C4 = (4096, 128, 3072, 8)        # skewed routing over many experts


def _case(name, kind, layer, T, routing="uniform"):
    K, E, N, top_k = layer
    return {"name": name, "kind": kind, "K": K, "E": E, "N": N, "top_k": top_k, "T": T, "routing": routing}


def listed():
    return [
        # one token of one request: latency, launches and host work
        _case("decode1_bf16", "bf16", C2, 1),
        # a small decode batch: most of the weights are read for one or two rows each
        _case("decode16_bf16", "bf16", C2, 16),
        _case("decode16_mxfp8", "mxfp8", C2, 16),
        # a large, odd decode batch: every expert is read for a handful of rows
        _case("decode131_bf16", "bf16", C2, 131),
        # a short prompt on a small layer
        _case("small256_bf16", "bf16", C0, 256),
        # prefill of a full batch, narrow experts (512 rows each)
        _case("prefill8192_bf16", "bf16", C2, 8192),
        # prefill of a ragged batch in mxfp8
        _case("prefill5003_mxfp8", "mxfp8", C2, 5003),
        # prefill, wide experts: tensor-bound, CTA pairs
        _case("wide4096_bf16", "bf16", C1, 4096),
        # the largest mxfp8 layer
        _case("large16384_mxfp8", "mxfp8", C3, 16384),
        # the largest call: skewed routing, hot and nearly empty experts
        _case("zipf65536_bf16", "bf16", C4, 65536, "zipf"),
        # training micro-batches: many narrow experts (pre-activations kept), few wide ones (recomputed)
        _case("train4099_bf16", "train", C2, 4099),
        _case("train4096_wide_bf16", "train", C1, 4096),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case: sizes log-uniform over the range of the listed ones, within their largest cost and memory."""
    while True:
        kind = rng.choice(["bf16", "bf16", "mxfp8", "train"])
        step = 256 if kind == "mxfp8" else 128
        K = max(1024, min(7168, step * round(_log_uniform(rng, 1024, 7168) / step)))
        N = max(512, min(28672, 256 * round(_log_uniform(rng, 512, 28672) / 256)))
        E = round(_log_uniform(rng, 8, 256))
        top_k = min(E, rng.randint(1, 8))
        T = round(_log_uniform(rng, 1, 65536)) if kind != "train" else round(_log_uniform(rng, 256, 32768))
        case = {"kind": kind, "K": K, "E": E, "N": N, "top_k": top_k, "T": T,
                "routing": rng.choice(["uniform", "uniform", "zipf"])}
        weights = 1.5 * E * N * K * (1 if kind == "mxfp8" else 2)
        rows = T * top_k * (K + N) * 2.0
        if weights > (11.5e9 if kind == "mxfp8" else 4e9) or rows > 8e9 or work(case)["flops"] > 1.5e13:
            continue
        if 3 * weights + rows > 60e9 or (kind == "train" and weights + rows > 8e9):
            continue
        return case


def _expected_experts(case):
    """Expected number of experts that receive a row."""
    E, k, T = case["E"], case["top_k"], case["T"]
    if case["routing"] == "uniform":
        share = [1.0 / E] * E
    else:
        w = [(e + 1) ** -1.2 for e in range(E)]
        share = [v / sum(w) for v in w]
    return sum(1.0 - (1.0 - min(1.0, k * p)) ** T for p in share)


def work(case):
    K, E, N, k, T = (case[n] for n in ("K", "E", "N", "top_k", "T"))
    elem = 1.0 + 1.0 / 32 if case["kind"] == "mxfp8" else 2.0
    weights = 1.5 * N * K
    if case["kind"] == "train":      # weights, x, d_out in; out, d_x, both weight gradients, routing-weight gradients out
        return {"bytes": 2.0 * (_expected_experts(case) + E) * weights + 4 * 2.0 * T * K + 8.0 * T * k,
                "flops": 9.0 * T * k * K * N}      # a recomputed gate/up GEMM is not counted
    return {"bytes": elem * _expected_experts(case) * weights + 2 * 2.0 * T * K + 4.0 * T * E,
            "flops": 3.0 * T * k * K * N}


def tolerance(case):
    # bf16 (or MX) activations between the two GEMMs, and the top_k results of a token summed in bf16 in any order.
    # Measured on the C0 and C2 layers at T = 1 ... 8192: 2.6e-3 ... 4.4e-3 (largest difference 1.6e-2 ... 4.3e-2)
    # against the same layer in 64 bits, up to 4.9e-3 (3.4e-2) between two runs; four times that is allowed.
    return {"rel": 0.018, "max": 0.18}


def _logits(case, g, dev):
    T, E = case["T"], case["E"]
    if case["routing"] == "uniform":
        return torch.randn(T, E, device=dev, generator=g)
    u = torch.rand(T, E, device=dev, generator=g).clamp_(1e-7, 1.0 - 1e-7)
    prior = -1.2 * torch.log(torch.arange(1, E + 1, device=dev, dtype=torch.float32))
    return prior - torch.log(-torch.log(u))      # Gumbel noise: the top_k are a sample without replacement


def _weights(g, dev, E, rows, cols):
    return torch.randn(E, rows, cols, device=dev, generator=g, dtype=torch.bfloat16).mul_(cols ** -0.5)


def _mx_weights(g, dev, E, rows, cols):
    """A quantised weight tensor and its blocked scales, a few experts at a time."""
    q = torch.empty(E, rows, cols, device=dev, dtype=torch.float8_e4m3fn)
    scales = torch.empty(E, rows * cols // 32, device=dev, dtype=torch.float8_e8m0fnu)
    step = max(1, int(1e9) // (rows * cols))
    for e in range(0, E, step):
        n = min(step, E - e)
        qe, se = P.quantize_mx(_weights(g, dev, n, rows, cols).view(n * rows, cols))
        q[e:e + n].view(torch.uint8).copy_(qe.view(torch.uint8).view(n, rows, cols))
        packed = P.pack_scales_blocked(se.view(torch.uint8).view(n, rows, cols // 32))
        scales[e:e + n].view(torch.uint8).copy_(packed.view(torch.uint8))
    return q, scales


def prepare(case, seed):
    dev = torch.device("cuda")
    K, E, N, k, T = (case[n] for n in ("K", "E", "N", "top_k", "T"))
    g = torch.Generator(device=dev).manual_seed(seed)
    s = {"kind": case["kind"], "top_k": k, "bpc": 2 if case["kind"] != "mxfp8" and N >= 8192 else 1,
         "x": torch.randn(T, K, device=dev, generator=g, dtype=torch.bfloat16), "logits": _logits(case, g, dev)}
    if case["kind"] == "mxfp8":
        s["w1"], s["w1_scales"] = _mx_weights(g, dev, E, N, K)
        s["w2"], s["w2_scales"] = _mx_weights(g, dev, E, K, N // 2)
    else:
        s["w1"] = _weights(g, dev, E, N, K)
        s["w2"] = _weights(g, dev, E, K, N // 2)
    if case["kind"] == "train":
        values, s["ids"] = torch.topk(s["logits"], k, dim=-1)
        s["ids"] = s["ids"].to(torch.int32).contiguous()
        s["wts"] = torch.softmax(values, -1).requires_grad_(True)
        s["recompute"] = N >= 8192 or T * k < 256 * E
        s["d_out"] = torch.randn(T, K, device=dev, generator=g, dtype=torch.bfloat16)
        for name in ("x", "w1", "w2"):
            s[name].requires_grad_(True)
    else:
        s["out"] = torch.empty(T, K, device=dev, dtype=torch.bfloat16)
    return s


def run(s):
    k = s["top_k"]
    if s["kind"] == "train":
        leaves = [s["x"], s["w1"], s["w2"], s["wts"]]
        out = P.moe_ffn(s["x"], s["w1"], s["w2"], s["ids"], s["wts"], recompute=s["recompute"])
        return [out.detach(), *torch.autograd.grad(out, leaves, s["d_out"])]
    _, wts, sorted_ids, expert_ids, npp = P.route_topk_align(s["logits"], k, bpc=s["bpc"])
    if s["kind"] == "bf16":
        return P.fused_moe_bf16(s["x"], s["w1"], s["w2"], sorted_ids, expert_ids, npp, wts, s["out"], k,
                                128, 64, 4, 4, s["bpc"])
    xq, xs = P.quantize_mx(s["x"])
    return P.fused_moe_mxfp8(xq, xs, s["w1"], s["w1_scales"], s["w2"], s["w2_scales"], sorted_ids, expert_ids, npp, wts,
                             s["out"], k, 128, 64, 4, 4)
