"""Performance cases of the quantized decode-projection path, through its public entry points.

Six kinds of pass, each a call (or short chain of calls) that a serving program makes:

  linear    tk.decode_linear_epilogue: one packed projection of M rows with its fused epilogue and,
            where asked for, the requantised output (decode M = 1 .. 16, chunks of a prefill above)
  mlp       the feed-forward block: tk.decode_swiglu, then the down projection with the residual
  lm_head   tk.lm_head_sample over a packed vocabulary head (argmax / categorical / top-k / top-p)
  stack     parallel.TPDecodeStack.forward on one GPU: consecutive decoder blocks' projections
  base_q    tk.base_qgemv / tk.base_qgemm over separate code / scale / bias planes
  seam      the two norm / activation -> quantiser seams of a block: tk.rms_norm_add* and
            tk.silu_mul_quant*

Weights are seeded Gaussians (sigma 0.02) quantised on the GPU by the rule of their format, activations
are unit Gaussians.  A state holds what a serving program keeps: packed weights and the step's input.
"""
from __future__ import annotations

import math

import torch

from quixicore_metal_b200 import parallel, tk, tk_torch

# columns and bytes of one block
BLOCK = {"q4_0": (32, 18), "q8_0": (32, 34), "q6_K": (256, 210), "mxfp8": (32, 33), "nvfp4": (16, 9), "mxfp4": (32, 17)}
DTYPE = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
SIZE = {"bf16": 2, "f16": 2, "f32": 4}


# ---- the cases -----------------------------------------------------------------------------------------
def listed():
    return [
        # one projection of an 8B-class block for one sequence: the smallest ordinary call, bound by latency
        # and by what the host does around the launch
        {"name": "linear_q4_0_4096_m1", "kind": "linear", "fmt": "q4_0", "M": 1, "K": 4096, "N": 4096, "dtype": "bf16",
         "activation": "none", "bias": True, "residual": False, "quant": "none"},
        # the shape of the reference project's published latencies: fp32 in and out, the whole epilogue
        {"name": "linear_q4_0_f32_m1", "kind": "linear", "fmt": "q4_0", "M": 1, "K": 1536, "N": 4096, "dtype": "f32",
         "activation": "silu", "bias": True, "residual": True, "quant": "none"},
        # feed-forward block of an 8B-class model, a few sequences at once
        {"name": "mlp_q6_K_m4", "kind": "mlp", "fmt": "q6_K", "M": 4, "K": 4096, "N": 14336, "dtype": "bf16"},
        # up projection of a 70B-class block, one sequence, output requantised for the next operator
        {"name": "linear_nvfp4_8192_m1", "kind": "linear", "fmt": "nvfp4", "M": 1, "K": 8192, "N": 28672, "dtype": "bf16",
         "activation": "none", "bias": True, "residual": False, "quant": "mxfp8"},
        # the same projection for a full batch or a prefill chunk: a real contraction
        {"name": "linear_mxfp4_8192_m256", "kind": "linear", "fmt": "mxfp4", "M": 256, "K": 8192, "N": 28672, "dtype": "bf16",
         "activation": "none", "bias": True, "residual": False, "quant": "mxfp8"},
        # greedy decoding of one sequence over a 128K vocabulary
        {"name": "lm_head_q8_0_t1_argmax", "kind": "lm_head", "fmt": "q8_0", "M": 1, "K": 4096, "N": 128256, "dtype": "bf16",
         "mode": "argmax", "k": 0},
        # a few sequences over a 32K vocabulary whose size is no multiple of anything
        {"name": "lm_head_q4_0_t7_topk", "kind": "lm_head", "fmt": "q4_0", "M": 7, "K": 4096, "N": 32003, "dtype": "bf16",
         "mode": "topk", "k": 8},
        # nucleus sampling of a full batch over a 128K vocabulary
        {"name": "lm_head_q8_0_t64_topp", "kind": "lm_head", "fmt": "q8_0", "M": 64, "K": 4096, "N": 128256, "dtype": "bf16",
         "mode": "topp", "k": 32},
        # four 70B-class blocks of a decode step: one sequence, and a batch of 32
        {"name": "stack_nvfp4_m1", "kind": "stack", "fmt": "nvfp4", "M": 1, "K": 8192, "N": 28672, "kv": 1024, "layers": 4,
         "dtype": "bf16"},
        {"name": "stack_nvfp4_m32", "kind": "stack", "fmt": "nvfp4", "M": 32, "K": 8192, "N": 28672, "kv": 1024, "layers": 4,
         "dtype": "bf16"},
        # a projection over separate planes, 4-bit codes with a scale and a bias per 32 columns
        {"name": "base_q4_g32_m1", "kind": "base_q", "bits": 4, "group": 32, "symmetric": False, "M": 1, "K": 8192, "N": 28672,
         "dtype": "bf16"},
        # the quantising seams of a prefill chunk of 4096 tokens
        {"name": "seam_fp8_4096", "kind": "seam", "M": 4096, "K": 8192, "quant": "fp8", "dtype": "bf16"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _log_mult(rng, lo, hi, unit):
    return max(1, round(_log_int(rng, lo, hi) / unit)) * unit


def draw(rng):
    """One case of the ranges above.  K is a multiple of 256 (hidden sizes are), N and M are anything;
    16-bit activations are the rule, fp32 ones (small batches) the exception."""
    kind = rng.choice(["linear"] * 5 + ["mlp"] + ["lm_head"] * 3 + ["stack", "base_q", "seam"])
    fmt = rng.choice(sorted(BLOCK))
    dtype = rng.choice(["bf16"] * 7 + ["f16"] * 2 + ["f32"])
    half = dtype if dtype != "f32" else "bf16"
    if kind == "linear":
        K = _log_mult(rng, 1024, 8192, 256)
        quant = rng.choice(["none", "none", "mxfp8", "fp8", "int8"])
        N = _log_mult(rng, 512, 28672, 32) if quant == "mxfp8" or rng.random() < 0.5 else _log_int(rng, 512, 28672)
        return {"kind": kind, "fmt": fmt, "M": _log_int(rng, 1, 8 if dtype == "f32" else 256), "K": K, "N": N, "dtype": dtype,
                "activation": rng.choice(["none", "none", "silu", "gelu"]), "bias": rng.random() < 0.5,
                "residual": rng.random() < 0.5, "quant": quant}
    if kind == "mlp":
        return {"kind": kind, "fmt": fmt, "M": _log_int(rng, 1, 64), "K": _log_mult(rng, 1024, 8192, 256),
                "N": _log_mult(rng, 2048, 14336, 256), "dtype": half}
    if kind == "lm_head":
        mode = rng.choice(["argmax", "categorical", "topk", "topp"])
        return {"kind": kind, "fmt": fmt, "M": _log_int(rng, 1, 64), "K": _log_mult(rng, 1024, 4096, 256),
                "N": _log_int(rng, 16000, 128256), "dtype": half, "mode": mode,
                "k": rng.randint(1, 64) if mode in ("topk", "topp") else 0}
    if kind == "stack":
        return {"kind": kind, "fmt": fmt, "M": _log_int(rng, 1, 32), "K": _log_mult(rng, 2048, 8192, 1024),
                "N": _log_mult(rng, 4096, 28672, 1024), "kv": 1024, "layers": rng.randint(1, 4), "dtype": half}
    if kind == "base_q":
        return {"kind": kind, "bits": rng.choice([2, 3, 4, 4, 5, 6, 8]), "group": rng.choice([32, 64, 128]),
                "symmetric": rng.random() < 0.5, "M": _log_int(rng, 1, 16), "K": _log_mult(rng, 1024, 8192, 256),
                "N": _log_int(rng, 1024, 28672), "dtype": half}
    return {"kind": kind, "M": _log_int(rng, 1, 4096), "K": _log_mult(rng, 1024, 8192, 256),
            "quant": rng.choice(["fp8", "int8", "block"]), "dtype": half}


# ---- packed weights ------------------------------------------------------------------------------------
def _halves(codes):
    """4-bit codes (..., n) -> bytes (..., n / 2): byte i holds code i (low) and code i + n / 2 (high)."""
    n = codes.shape[-1] // 2
    return codes[..., :n] | (codes[..., n:] << 4)


def _f16_bytes(d):
    return d.to(torch.float16).unsqueeze(-1).view(torch.uint8)


def _e4m3(v):
    return v.clamp(-448.0, 448.0).to(torch.float8_e4m3fn)


def _e2m1(v):
    steps = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=v.device)
    code = torch.bucketize(v.abs(), steps, out_int32=True).to(torch.uint8)
    return code | ((v < 0).to(torch.uint8) << 3)


def _pack_rows(fmt, W):
    """fp32 (rows, K) -> packed blocks uint8 (rows, K / block, block_bytes)."""
    bk, bb = BLOCK[fmt]
    rows, K = W.shape
    B = W.view(rows, K // bk, bk)
    out = torch.empty((rows, K // bk, bb), dtype=torch.uint8, device=W.device)
    amax = B.abs().amax(-1)
    if fmt == "q8_0":
        d = (amax / 127.0).half().float()
        out[..., :2] = _f16_bytes(d)
        out[..., 2:] = (B / d.clamp_min(1e-30)[..., None]).round_().clamp_(-127, 127).to(torch.int8).view(torch.uint8)
    elif fmt == "q4_0":
        d = (torch.gather(B, -1, B.abs().argmax(-1, keepdim=True))[..., 0] / -8.0).half().float()
        safe = torch.where(d == 0, torch.ones_like(d), d)
        out[..., :2] = _f16_bytes(d)
        out[..., 2:] = _halves((B / safe[..., None]).round_().add_(8).clamp_(0, 15).to(torch.uint8))
    elif fmt == "q6_K":
        sub = B.view(rows, K // bk, 16, 16)
        smax = sub.abs().amax(-1) / 31.0
        d = (smax.amax(-1) / 127.0).half().float().clamp_min(2.0 ** -24)
        sc = (smax / d[..., None]).round_().clamp_(1, 127)
        q = (sub / (d[..., None] * sc)[..., None]).round_().clamp_(-32, 31).add_(32).to(torch.uint8)
        q = q.view(rows, K // bk, 2, 4, 32)                      # 128-column half, 32-column quarter, column
        lo, hi = q & 15, q >> 4
        out[..., :128] = torch.cat([lo[:, :, :, :2] | (lo[:, :, :, 2:] << 4)], -1).reshape(rows, K // bk, 128)
        out[..., 128:192] = (hi[:, :, :, 0] | (hi[:, :, :, 1] << 2) | (hi[:, :, :, 2] << 4) | (hi[:, :, :, 3] << 6)).reshape(rows, K // bk, 64)
        out[..., 192:208] = sc.to(torch.int8).view(torch.uint8)
        out[..., 208:] = _f16_bytes(d)
    elif fmt == "nvfp4":
        s = _e4m3(amax / 6.0)
        out[..., 0] = s.view(torch.uint8)
        out[..., 1:] = _halves(_e2m1(B / s.float().clamp_min(2.0 ** -9)[..., None]))
    else:
        e = torch.ceil(torch.log2(amax.clamp_min(1e-30) / (448.0 if fmt == "mxfp8" else 6.0)))
        scaled = B * torch.exp2(-e)[..., None]
        out[..., 0] = (e + 127).to(torch.uint8)
        out[..., 1:] = _e4m3(scaled).view(torch.uint8) if fmt == "mxfp8" else _halves(_e2m1(scaled))
    return out


def _weights(fmt, N, K, gen):
    bk, bb = BLOCK[fmt]
    out = torch.empty((N, K // bk, bb), dtype=torch.uint8, device="cuda")
    step = max(1, (1 << 26) // K)
    for r in range(0, N, step):
        n = min(step, N - r)
        out[r:r + n] = _pack_rows(fmt, torch.randn((n, K), generator=gen, device="cuda").mul_(0.02))
    return out


def _packed_bytes(fmt, N, K):
    bk, bb = BLOCK[fmt]
    return N * (K // bk) * bb


# ---- a case's state, pass, work and tolerance ----------------------------------------------------------
def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    dt = DTYPE[case["dtype"]]
    M, K = case["M"], case["K"]

    def rand(*shape):
        return torch.randn(shape, generator=gen, device="cuda").to(dt)

    s = {"case": case, "seed": seed & 0x7FFFFFFF}
    kind = case["kind"]
    if kind == "seam":
        s.update(x=rand(M, K), residual=rand(M, K), gate=rand(M, K), weight=(1 + 0.1 * torch.randn(K, generator=gen, device="cuda")).to(dt))
        return s
    N = case["N"]
    if kind == "linear":
        s.update(x=rand(M, K), w=_weights(case["fmt"], N, K, gen), bias=rand(N) * 0.01 if case["bias"] else None,
                 residual=rand(M, N) if case["residual"] else None)
    elif kind == "mlp":
        s.update(x=rand(M, K), gate=_weights(case["fmt"], N, K, gen), up=_weights(case["fmt"], N, K, gen),
                 down=_weights(case["fmt"], K, N, gen), residual=rand(M, K))
    elif kind == "lm_head":
        s.update(h=rand(M, K), w=_weights(case["fmt"], N, K, gen))
    elif kind == "stack":
        fmt, kv = case["fmt"], case["kv"]
        layers = [{"qkv": _weights(fmt, K + 2 * kv, K, gen), "o": _weights(fmt, K, K, gen), "gate": _weights(fmt, N, K, gen),
                   "up": _weights(fmt, N, K, gen), "down": _weights(fmt, K, N, gen)} for _ in range(case["layers"])]
        # no norms in between: a small input keeps the residual stream of four blocks of ordinary size
        s.update(x=rand(M, K) * 0.05, stack=parallel.TPDecodeStack(layers, fmt))
    else:
        bits, group = case["bits"], case["group"]
        span = 2 ** bits - 1
        scale = (0.1 + 0.02 * torch.rand((N, K // group), generator=gen, device="cuda")) / span
        s.update(x=rand(K, M), codes=torch.randint(0, 256, (N, K * bits // 8), dtype=torch.uint8, generator=gen, device="cuda"),
                 scales=scale.bfloat16(), biases=None if case["symmetric"] else (scale * (-0.5 * span)).bfloat16())
    return s


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "linear":
        if c["quant"] == "none":
            return tk.decode_linear_epilogue(state["x"], state["w"], state["bias"], state["residual"],
                                             activation=c["activation"], format=c["fmt"])
        return tk.decode_linear_epilogue(state["x"], state["w"], state["bias"], state["residual"],
                                         activation=c["activation"], format=c["fmt"], output_quant=c["quant"])
    if kind == "mlp":
        mid = tk.decode_swiglu(state["x"], state["gate"], state["up"], format=c["fmt"])
        return mid, tk.decode_linear_epilogue(mid, state["down"], None, state["residual"], format=c["fmt"])
    if kind == "lm_head":
        return tk.lm_head_sample(state["h"], state["w"], mode=c["mode"], k=c["k"], temperature=0.8, seed=state["seed"],
                                 format=c["fmt"], top_p=0.9)
    if kind == "stack":
        return state["stack"].forward(state["x"])
    if kind == "base_q":
        call = tk.base_qgemv if c["M"] == 1 else tk.base_qgemm
        return call(state["codes"], state["scales"], state["biases"], state["x"], c["bits"], c["group"], "bf16",
                    symmetric=c["symmetric"])
    x, residual, weight, gate = state["x"], state["residual"], state["weight"], state["gate"]
    if c["quant"] == "fp8":
        return tk.rms_norm_add_fp8(x, residual, weight), tk.silu_mul_quant_fp8(x, gate)
    if c["quant"] == "int8":
        return tk_torch.rms_norm_add_int8_dyn(x, residual, weight), tk.silu_mul_quant_int8(x, gate)
    return tk.rms_norm_add_per_block(x, residual, weight), tk.silu_mul_quant_fp8_group(x, gate)


def work(case):
    kind, M, K, es = case["kind"], case["M"], case["K"], SIZE[case["dtype"]]
    if kind == "seam":
        scales = (2 if case["quant"] != "block" else 2 * (K // 128)) * 4 * M
        return {"bytes": M * K * (es * 4 + es + 2) + K * es + scales, "flops": 12 * M * K}
    N = case["N"]
    if kind == "base_q":
        planes = N * K * case["bits"] // 8 + N * (K // case["group"]) * 2 * (1 if case["symmetric"] else 2)
        return {"bytes": planes + es * M * (K + N), "flops": 2 * M * N * K}
    if kind == "lm_head":
        return {"bytes": _packed_bytes(case["fmt"], N, K) + es * M * K + 4 * M, "flops": 2 * M * N * K}
    if kind == "mlp":
        return {"bytes": 2 * _packed_bytes(case["fmt"], N, K) + _packed_bytes(case["fmt"], K, N) + es * M * (3 * K + N),
                "flops": 6 * M * N * K}
    if kind == "stack":
        one = sum(_packed_bytes(case["fmt"], n, k) for n, k in ((K + 2 * case["kv"], K), (K, K), (N, K), (N, K), (K, N)))
        flops = 2 * M * ((2 * K + 2 * case["kv"]) * K + 3 * N * K)
        return {"bytes": case["layers"] * one + 2 * es * M * K, "flops": case["layers"] * flops}
    out = {"none": es, "mxfp8": 33 / 32, "fp8": 1, "int8": 1}[case["quant"]] * M * N + (4 * M if case["quant"] in ("fp8", "int8") else 0)
    ins = es * (M * K + (N if case["bias"] else 0) + (M * N if case["residual"] else 0))
    return {"bytes": _packed_bytes(case["fmt"], N, K) + ins + out, "flops": 2 * M * N * K}


def tolerance(case):
    """fp32 sums in any order, one rounding to the output type: a few outputs land on the other side of a
    rounding boundary (one unit of the last place), and of the codes made from them a few.  Token ids are
    whole: the same draw from the same logits."""
    kind = case["kind"]
    if kind == "lm_head":
        return "exact"
    rel = {"bf16": 2e-3, "f16": 3e-4, "f32": 1e-5}[case["dtype"]]
    if kind == "stack":
        return {"rel": 5 * rel, "max": 0.1}               # the flips of one block feed the next
    if kind == "mlp":
        return {"rel": 2 * rel, "max": 0.02}
    if kind == "seam":
        return {"rel": 1e-5, "max": 0.01, "differ": 1e-3}
    return {"rel": rel, "max": 10 * rel, "differ": 5e-3}
