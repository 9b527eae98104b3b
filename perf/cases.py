"""Performance cases of the framework's two hot paths, through the entry points a user's program calls.

Kinds of case:
  gemm      `gemm.custom_kernel` on K-major e4m3fn operands (block scales uniform in [0.5, 2] * 2^-7)
  gemm_ref  `gemm.custom_kernel` on the reference generator's own tuple: transposed views of [k, m] / [k, n]
            e4m3fnuz tensors with signed N(0, 1) scales; with "amax" the operands are block-quantised to +-240
  moe       `moe.custom_kernel`: router, top-k, routed and shared experts in one call
  moe_topk  `moe.moe_forward` with the router logits given (`run_topk`): every stage tensor is an output
  moe_ep    `multi_gpu.ExpertParallelMoE.forward`, the expert-parallel layer, on one GPU, with Zipf-skewed routing
"""
import math

import numpy as np
import torch

from radeonflow_kernels_b200 import gemm, moe, multi_gpu

DEV = "cuda:0"
BLOCK = 128
ZIPF_S = 1.1


def listed():
    return [
        # A projection over a 1024-token batch with a short K: the shortest of the sweep's shapes, bound by launch
        # and set-up latency.
        {"name": "gemm_1024x4096x512", "kind": "gemm", "m": 1024, "n": 4096, "k": 512},
        # A few sequences in decode: hardly any rows, a narrow output (N = 576 ends in half a scale block), a long K.
        {"name": "gemm_64x576x7168", "kind": "gemm", "m": 64, "n": 576, "k": 7168},
        # The sweep's headline small shape: too few tiles for the chip, a long K.
        {"name": "gemm_1024x1536x7168", "kind": "gemm", "m": 1024, "n": 1536, "k": 7168},
        # Ragged in every direction: rows that end inside a tile, a last column block of one half.
        {"name": "gemm_1337x3008x1920", "kind": "gemm", "m": 1337, "n": 3008, "k": 1920},
        # Prefill, middle K: the per-tile cost counts as much as the K loop.
        {"name": "gemm_6144x7168x2048", "kind": "gemm", "m": 6144, "n": 7168, "k": 2048},
        # Prefill, long K: the sweep's largest shape.
        {"name": "gemm_6144x4608x7168", "kind": "gemm", "m": 6144, "n": 4608, "k": 7168},
        # The N-split configuration's whole GEMM on one GPU.
        {"name": "gemm_16384x28672x7168", "kind": "gemm", "m": 16384, "n": 28672, "k": 7168},
        # A user of the reference who hands over its generator's tensors as they are (layout and FP8 format).
        {"name": "gemm_ref_1024x7168x2048", "kind": "gemm_ref", "m": 1024, "n": 7168, "k": 2048, "amax": False},
        # One decode step of a batch of 128 sequences: every expert's weights for a few rows each.
        {"name": "moe_t128_e32", "kind": "moe", "t": 128, "d": 7168, "f": 2048, "e": 32, "k": 4},
        # A ragged prefill chunk through the reference's C entry, logits given, stage tensors out.
        {"name": "moe_topk_t1111_e32", "kind": "moe_topk", "t": 1111, "d": 7168, "f": 2048, "e": 32, "k": 4},
        # The single-GPU layer of the benchmark.
        {"name": "moe_t8192_e32", "kind": "moe", "t": 8192, "d": 7168, "f": 2048, "e": 32, "k": 4},
        # The expert-parallel layer of the benchmark, all 256 experts on one GPU.
        {"name": "moe_ep_t32768_e256", "kind": "moe_ep", "t": 32768, "d": 7168, "f": 2048, "e": 256, "k": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: GEMMs over M = 1..8192 (any M; multiples of 16 in the reference's layout), N = 64..7168,
    K = 128..7168; layers over 16..8192 tokens, 4 to 64 experts, top-2 to top-8."""
    kind = rng.choice(["gemm", "gemm", "gemm", "gemm_ref", "moe", "moe", "moe_topk", "moe_ep"])
    if kind in ("gemm", "gemm_ref"):
        m = _log_int(rng, 1, 8192)
        n = 64 * _log_int(rng, 1, 112)
        k = 128 * _log_int(rng, 1, 56)
        if kind == "gemm":
            return {"kind": kind, "m": m, "n": n, "k": k}
        return {"kind": kind, "m": 16 * ((m + 15) // 16), "n": n, "k": k, "amax": rng.random() < 0.5}
    t = _log_int(rng, 16, 8192)
    e = rng.choice([4, 8, 32, 64])
    k = rng.choice([2, 4, 8]) if e >= 8 else rng.choice([2, 4])
    d, f = rng.choice([(7168, 2048), (7168, 2048), (4096, 1536), (1024, 512)])
    return {"kind": kind, "t": t, "d": d, "f": f, "e": e, "k": k}


# ------------------------------------------------------------------------------------------------ inputs --
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _prepare_gemm(case, g):
    m, n, k = case["m"], case["n"], case["k"]
    kb, nb = k // BLOCK, (n + BLOCK - 1) // BLOCK

    def fp8(rows):
        return torch.randn(rows, k, generator=g, device=DEV).clamp_(-240, 240).to(torch.float8_e4m3fn)

    def scales(rows):
        return (0.5 + 1.5 * torch.rand(rows, kb, generator=g, device=DEV)) * 2.0 ** -7

    return {"data": (fp8(m), fp8(n), scales(m), scales(nb), torch.empty(m, n, dtype=torch.bfloat16, device=DEV))}


def _prepare_gemm_ref(case, g):
    m, n, k = case["m"], case["n"], case["k"]
    kb, nb = k // BLOCK, (n + BLOCK - 1) // BLOCK

    def randn(*shape):
        return torch.randn(*shape, generator=g, device=DEV)

    a, b = randn(k, m), randn(k, n)
    if case["amax"]:
        # block quantisation: each 1 x 128 group of A and 128 x 128 block of B is scaled to its own largest magnitude
        sa = a.view(kb, BLOCK, m).abs().amax(1) / 240.0
        a = a / sa.repeat_interleave(BLOCK, 0)
        pad = torch.nn.functional.pad(b, (0, nb * BLOCK - n)).view(kb, BLOCK, nb, BLOCK)
        sb = pad.abs().amax((1, 3)) / 240.0
        b = b / sb.repeat_interleave(BLOCK, 0).repeat_interleave(BLOCK, 1)[:, :n]
    else:
        sa, sb = randn(kb, m), randn(kb, nb)
    a8 = a.clamp_(-240, 240).to(torch.float8_e4m3fnuz)
    b8 = b.clamp_(-240, 240).to(torch.float8_e4m3fnuz)
    c = torch.empty(m, n, dtype=torch.bfloat16, device=DEV)
    return {"data": (a8.t(), b8.t(), sa.contiguous().t(), sb.contiguous().t(), c)}


def _layer_weights(case, g):
    """The reference generator's distributions: router N(0, 1/d), gate and up N(0, 1/f), down N(0, 1/d)."""
    d, f, e = case["d"], case["f"], case["e"]

    def randn(rows, cols, fan):
        return torch.randn(rows, cols, generator=g, device=DEV, dtype=torch.float16).mul_(1.0 / math.sqrt(fan))

    w = {"router.weight": randn(e, d, d)}
    for i in range(e):
        for j, (rows, cols, fan) in enumerate(((d, f, f), (d, f, f), (f, d, d))):
            w[f"experts.{i}.{j}.weight"] = randn(rows, cols, fan)
    for j, (rows, cols, fan) in enumerate(((d, f, f), (d, f, f), (f, d, d))):
        w[f"shared_experts.{j}.weight"] = randn(rows, cols, fan)
    return w


def _prepare_layer(case, g):
    x = torch.randn(1, case["t"], case["d"], generator=g, device=DEV, dtype=torch.float16)
    config = {"d_hidden": case["d"], "d_expert": case["f"], "n_routed_experts": case["e"], "n_shared_experts": 1,
              "n_experts_per_token": case["k"], "batch_size": 1, "seq_len": case["t"]}
    return {"x": x, "weights": _layer_weights(case, g), "config": config}


class _Layer:
    """Gives the expert-parallel object's buffers back with the state that holds it."""

    def __init__(self, *args, **kwargs):
        self.moe = multi_gpu.ExpertParallelMoE(*args, **kwargs)

    def __del__(self):
        if hasattr(self, "moe"):
            self.moe.close()


def prepare(case, seed):
    g = _gen(seed)
    if case["kind"] == "gemm":
        return dict(_prepare_gemm(case, g), kind="gemm")
    if case["kind"] == "gemm_ref":
        return dict(_prepare_gemm_ref(case, g), kind="gemm_ref")
    s = dict(_prepare_layer(case, g), kind=case["kind"])
    if case["kind"] == "moe_topk":
        s["scores"] = (s["x"][0] @ s["weights"]["router.weight"].t()).contiguous()
    elif case["kind"] == "moe_ep":
        rank = np.random.default_rng(seed).permutation(case["e"])
        bias = torch.from_numpy((-ZIPF_S * np.log1p(rank.astype(np.float64))).astype(np.float32)).to(DEV)
        s["layer"] = _Layer(s["config"], s["weights"], case["t"], DEV, router_bias=bias)
    return s


# ------------------------------------------------------------------------------------------------ one pass --
def run(state):
    kind = state["kind"]
    if kind in ("gemm", "gemm_ref"):
        return gemm.custom_kernel(state["data"])
    if kind == "moe":
        return moe.custom_kernel((state["x"], state["weights"], state["config"]))
    if kind == "moe_topk":
        _, buffers = moe.moe_forward(state["x"], state["weights"], state["config"], expert_scores=state["scores"])
        return buffers.stages
    return state["layer"].moe.forward(state["x"][0])


def work(case):
    if case["kind"] in ("gemm", "gemm_ref"):
        m, n, k = case["m"], case["n"], case["k"]
        kb, nb = k // BLOCK, (n + BLOCK - 1) // BLOCK
        return {"bytes": m * k + n * k + 4 * (m + nb) * kb + 2 * m * n, "flops": 2.0 * m * n * k}
    t, d, f, e, k = (case[q] for q in "tdfek")
    flops = 2.0 * 3 * d * f * (t * k + t) + 2.0 * t * e * d
    # weights of every expert that can be hit, the shared expert and the router; tokens in and out
    nbytes = 2.0 * (3 * d * f * (min(e, t * k) + 1) + e * d + 2 * t * d)
    if case["kind"] == "moe_topk":
        # no router GEMM; the logits come in, and every stage tensor is an output
        flops -= 2.0 * t * e * d
        nbytes += 2.0 * (t * e - e * d) + 2.0 * (t * k * (2 * d + f) + t * (f + d)) + 24.0 * t * k
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] in ("gemm", "gemm_ref"):
        # Against a 64-bit computation every size shows 1.7e-3 (the bf16 rounding of the result) with single values
        # off by 4e-3; two fp32 summation orders differ by 3e-5 and by one bf16 step (8e-3) of single values.
        return {"rel": 4e-3, "max": 3e-2}
    if case["kind"] == "moe_topk":
        # Logits given: 5e-4 against a 64-bit computation (fp16 roundings between the stages), no index differs.
        return {"rel": 2e-3, "max": 1.2e-2, "differ": 0.0}
    # With the router inside, sums in another order round single fp16 logits the other way, and of 8192 tokens one or
    # two then choose another last expert: 8e-4 over the whole output, 0.3 within such a token's row.
    return {"rel": 4e-3, "max": 0.8}
