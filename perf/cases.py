"""The workloads this package is timed on: attention calls as a model's forward or training step makes them.

A case is a dict of plain values:
    op      "rope"   fused-RoPE attention with the caller's cos / sin tables
            "theta"  the same with the tables formed on the device from the base theta
            "flash"  plain attention with grouped K / V heads
            "corope" Co-RoPE attention with grouped K / V heads
    train   False: forward only (prefill, evaluation).  True: forward and backward (a training step's attention)
    B, Hq, Hkv, N, D, dtype, causal
    layout  "bhnd": contiguous [B, H, N, D] tensors.  "bnhd": [B, N, H, D] buffers viewed as [B, H, N, D], as the
            projections of a transformer layer leave them
One pass is one call of the public entry point, and for `train` the gradients of q, k and v through autograd.
"""

import math

import torch

import corope_b200

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
THETA = 10000.0


def _case(name, op, train, B, Hq, Hkv, N, D, dtype, causal=True, layout="bhnd"):
    return {"name": name, "op": op, "train": train, "B": B, "Hq": Hq, "Hkv": Hkv, "N": N, "D": D, "dtype": dtype, "causal": causal, "layout": layout}


def listed():
    return [
        # the smallest shape of the benchmark's sweep, forward only: what a call costs when there is little to compute
        _case("rope-512-d64-fwd", "rope", False, 4, 8, 8, 512, 64, "f16"),
        # fp32 at the same shape: the setting in which models are checked against their reference
        _case("rope-512-d64-fp32", "rope", True, 4, 8, 8, 512, 64, "f32"),
        # training steps at the shapes of the Llama-7B and Llama-70B rows of the benchmark; the first is its default workload
        _case("rope-7b-4k", "rope", True, 2, 32, 32, 4096, 128, "bf16"),
        _case("rope-70b-1k", "rope", True, 2, 64, 64, 1024, 128, "bf16"),
        # long-context training, the largest of all
        _case("rope-64k", "rope", True, 1, 8, 8, 65536, 128, "bf16"),
        # a small model's head dimension in a training step
        _case("rope-4k-d64", "rope", True, 2, 8, 8, 4096, 64, "f16"),
        # prefill of one prompt: a length that is no multiple of anything, buffers as the projections leave them
        _case("rope-prompt", "rope", False, 1, 32, 32, 1777, 128, "bf16", layout="bnhd"),
        # bidirectional training (an encoder) on sequences of 1000 tokens, angles from theta
        _case("theta-encoder-1000", "theta", True, 4, 16, 16, 1000, 64, "bf16", causal=False),
        # grouped K / V heads without rotation, training, buffers as the projections leave them
        _case("flash-gqa-4k", "flash", True, 1, 32, 8, 4096, 128, "bf16", layout="bnhd"),
        # Co-RoPE: a training step at the benchmark's shape, the fp32 check of a small model, prefill of a prompt
        _case("corope-gqa-2k", "corope", True, 2, 32, 8, 2048, 128, "bf16"),
        _case("corope-512-fp32", "corope", True, 1, 8, 2, 512, 64, "f32"),
        _case("corope-prompt", "corope", False, 1, 32, 8, 1500, 128, "f16", layout="bnhd"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the same kinds.  Lengths are log-uniform, half of them arbitrary and half multiples of 128; batch and
    head counts are cut down until the case costs no more than the listed ones of its kind."""
    op = rng.choice(("rope", "rope", "rope", "theta", "flash", "flash", "corope", "corope"))
    dtype = rng.choice(("bf16", "bf16", "bf16", "f16", "f16", "f32"))
    train = rng.random() < 0.6
    D = 128 if dtype != "f32" and rng.random() < 0.65 else rng.choice((64, 128))
    whole = rng.random() < 0.5   # a multiple of 128
    causal = op == "corope" or rng.random() < 0.8
    layout = rng.choice(("bhnd", "bnhd"))
    if op == "corope":
        longest = 4096 if dtype != "f32" else 1024
    else:
        longest = 2048 if dtype == "f32" else 65536 if whole else 6000
    N = _log_uniform(rng, 48, longest)
    if whole:
        N = max(128, N // 128 * 128)
    Hkv = rng.choice((1, 2, 4, 8, 16, 32)) if op in ("rope", "theta") else rng.choice((1, 2, 4, 8))
    G = 1 if op in ("rope", "theta") else rng.choice((1, 2, 3, 4, 4, 8))
    B = rng.choice((1, 1, 2, 4))
    if op == "corope":
        most = 2.1e9 if dtype != "f32" else 1.0e8           # (query, key, frequency) triples
        cost = N * N / 2 * D / 2
    else:
        most = 2.3e11 * D if whole and dtype != "f32" else 6.0e10   # operations
        cost = G * (4.0 * N * N * D * (0.5 if causal else 1.0)) * (3.5 if train else 1.0)
    while B > 1 and B * Hkv * cost > most:
        B //= 2
    while Hkv > 1 and B * Hkv * cost > most:
        Hkv //= 2
    while G > 1 and op == "flash" and B * Hkv * cost > most:
        G, cost = G // 2, cost / G * (G // 2)
    if B * Hkv * cost > most:   # even one head is too much
        N = int(N * (most / (B * Hkv * cost)) ** 0.5) // 128 * 128 - (0 if whole else 1)
    case = _case("", op, train, B, Hkv * G, Hkv, N, D, dtype, causal, layout)
    del case["name"]
    return case


def prepare(case, seed):
    """Inputs ~ N(0, 1), the benchmark's distribution, and the rotation tables that a model keeps next to its weights."""
    B, N, D, dtype = case["B"], case["N"], case["D"], DTYPES[case["dtype"]]
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def tensor(heads):
        if case["layout"] == "bnhd":
            return torch.randn((B, N, heads, D), generator=gen, device="cuda", dtype=dtype).transpose(1, 2)
        return torch.randn((B, heads, N, D), generator=gen, device="cuda", dtype=dtype)

    state = {"case": case, "scale": D ** -0.5}
    for name, heads in (("q", case["Hq"]), ("k", case["Hkv"]), ("v", case["Hkv"])):
        state[name] = tensor(heads).requires_grad_(case["train"])
    if case["train"]:
        state["do"] = tensor(case["Hq"])
    if case["op"] == "rope":
        freq = THETA ** (-torch.arange(0, D, 2, device="cuda", dtype=torch.float32) / D)
        angle = torch.outer(torch.arange(N, device="cuda", dtype=torch.float32), freq)
        state["cos"], state["sin"] = (torch.cat((t, t), dim=1) for t in (angle.cos(), angle.sin()))
    return state


def run(state):
    case, q, k, v = state["case"], state["q"], state["k"], state["v"]
    op, causal, scale = case["op"], case["causal"], state["scale"]
    if op == "rope":
        o = corope_b200.fused_rope_attention(q, k, v, causal, scale, state["cos"], state["sin"])
    elif op == "theta":
        o = corope_b200.fused_rope_attention_theta(q, k, v, causal, scale, THETA)
    elif op == "flash":
        o = corope_b200.flash_attention(q, k, v, causal, scale)
    else:
        o = corope_b200.corope_gqa_attention(q, k, v, causal, scale, THETA)
    if not case["train"]:
        return {"o": o}
    dq, dk, dv = torch.autograd.grad(o, (q, k, v), state["do"])
    return {"o": o.detach(), "dq": dq, "dk": dk, "dv": dv}


def work(case):
    """Tensors of the pass read or written once; the multiply-adds of the score and value products (two forward, five more
    backward), and for Co-RoPE those of the leader's scores (once forward, recomputed and differentiated backward)."""
    B, Hq, Hkv, N, D = (case[x] for x in ("B", "Hq", "Hkv", "N", "D"))
    e = 4 if case["dtype"] == "f32" else 2
    q_elems, kv_elems = B * Hq * N * D, B * Hkv * N * D
    pairs = N * N * (0.5 if case["causal"] else 1.0)
    nbytes = (2 * q_elems + 2 * kv_elems) * e           # q, o; k, v
    flops = 4.0 * B * Hq * pairs * D
    if case["train"]:
        nbytes += (2 * q_elems + 2 * kv_elems) * e      # dO, dq; dk, dv
        flops *= 3.5
    if case["op"] == "rope":
        nbytes += 2 * N * (D // 2) * 4
    if case["op"] == "corope":
        flops += 2.0 * B * Hkv * pairs * D * (4 if case["train"] else 1)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Relative 2-norm between two correct implementations at one precision.  16-bit: operands (rotated q and k, P, dS) and
    results are rounded to 8 (bf16) or 11 bits (f16).  fp32: sums of a few hundred terms; Co-RoPE phases reach some hundred
    radians, where one unit in the last place of the angle is 1.5e-5."""
    if case["dtype"] == "bf16":
        return {"rel": 1e-2}
    if case["dtype"] == "f16":
        return {"rel": 4e-3}
    return {"rel": 1e-4 if case["op"] == "corope" else 1e-5}
