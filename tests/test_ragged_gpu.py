"""Lengths that are not whole tiles, on the split-operand kernels: one key, one short of / one beyond the 64-row steps, the 128-row
blocks and the 256-row work items; both head dimensions, causal and full, with and without rotation, grouped heads, transposed
buffers.  Tolerances as in test_gpu_parity.py."""

import math
import os

import pytest
import torch

import oracle
from helpers import check16, draw, ext, pkg

pytestmark = pytest.mark.gpu

TOL_FWD_16, TOL_BWD_16 = 1e-2, 2e-2


def _label():
    return os.environ.get("PYTEST_CURRENT_TEST", "?").split("::")[-1].split(" ")[0]


def _check(outs, refs, dtype):
    check16(_label() + " O", outs[0], refs[0], TOL_FWD_16, dtype, strict=True)
    for name, got, ref in zip(("dQ", "dK", "dV"), outs[1:], refs[1:]):
        check16(_label() + " " + name, got, ref, TOL_BWD_16, dtype)


def _run(fn, q, k, v, do, *args):
    qd, kd, vd = (t.cuda().requires_grad_(True) for t in (q, k, v))
    o = fn(qd, kd, vd, *args)
    o.backward(do.cuda())
    ext.check_status()
    return tuple(t.detach().float().cpu() for t in (o, qd.grad, kd.grad, vd.grad))


@pytest.mark.parametrize("N", [1, 63, 65, 127, 129, 193, 255, 257, 449])
@pytest.mark.parametrize("D,causal,dtype", [(128, True, torch.bfloat16), (128, False, torch.float16), (64, True, torch.float16),
                                            (64, False, torch.bfloat16)])
def test_rope_at_tile_edges(N, D, causal, dtype):
    B, H = 1, 3
    q, k, v, do = (draw((B, H, N, D), 200 + i, dtype) for i in range(4))
    cos, sin = oracle.precompute_freqs_cis(D, N, 10000.0)
    s = D ** -0.5
    outs = _run(pkg.fused_rope_attention, q, k, v, do, causal, s, cos.cuda(), sin.cuda())
    refs = (oracle.rope_attn_fwd(q, k, v, causal, s, cos, sin),) + tuple(oracle.rope_attn_bwd(q, k, v, do, causal, s, cos, sin))
    _check(outs, refs, dtype)


@pytest.mark.parametrize("N,D,causal", [(200, 128, True), (300, 64, False), (1000, 64, True), (129, 128, False)])
def test_grouped_heads_in_transposed_buffers(N, D, causal):
    B, Hq, Hkv, dtype = 2, 6, 2, torch.bfloat16
    q, do = (draw((B, N, Hq, D), 210 + i, dtype).transpose(1, 2) for i in range(2))
    k, v = (draw((B, N, Hkv, D), 212 + i, dtype).transpose(1, 2) for i in range(2))
    s = D ** -0.5
    outs = _run(pkg.flash_attention, q, k, v, do, causal, s)
    refs = (oracle.attn_gqa_fwd(q, k, v, causal, s),) + tuple(oracle.attn_gqa_bwd(q, k, v, do, causal, s))
    _check(outs, refs, dtype)


@pytest.mark.parametrize("causal", [True, False])
def test_rows_of_the_next_head_are_not_seen(causal):
    # head 1 holds values 100 times as large (its V and dO even infinite in one element): head 0 must not change by a bit
    B, H, N, D, dtype = 1, 2, 200, 128, torch.bfloat16
    q, k, v, do = (draw((B, H, N, D), 220 + i, dtype) for i in range(4))
    base = _run(pkg.flash_attention, q, k, v, do, causal, D ** -0.5)
    for t in (q, k, v, do):
        t[:, 1] *= 100
    v[0, 1, 0, 0] = do[0, 1, 0, 0] = float("inf")
    outs = _run(pkg.flash_attention, q, k, v, do, causal, D ** -0.5)
    for a, b in zip(base, outs):   # every sum has one owner and one order
        assert torch.equal(a[:, 0], b[:, 0])


def test_theta_with_a_ragged_length():
    B, H, N, D, dtype = 2, 2, 333, 64, torch.bfloat16
    q, k, v, do = (draw((B, H, N, D), 230 + i, dtype) for i in range(4))
    cos, sin = oracle.precompute_freqs_cis(D, N, 10000.0)
    outs = _run(pkg.fused_rope_attention_theta, q, k, v, do, False, D ** -0.5, 10000.0)
    refs = (oracle.rope_attn_fwd(q, k, v, False, D ** -0.5, cos, sin),) + tuple(oracle.rope_attn_bwd(q, k, v, do, False, D ** -0.5, cos, sin))
    _check(outs, refs, dtype)


def _exact(q, k, v, do, causal, s, cos, sin):
    """The same in 64 bits: rotated attention and its gradients."""
    q, k, v = (t.cuda().double().requires_grad_(True) for t in (q, k, v))
    half = q.shape[-1] // 2
    c, sn = cos[:, :half].cuda().double(), sin[:, :half].cuda().double()
    qr, kr = (torch.cat((x[..., :half] * c - x[..., half:] * sn, x[..., half:] * c + x[..., :half] * sn), -1) for x in (q, k))
    w = qr @ kr.transpose(-1, -2) * s
    if causal:
        w = w.masked_fill(torch.ones_like(w, dtype=torch.bool).triu(1), float("-inf"))
    o = w.softmax(-1) @ v
    return (o.detach(),) + torch.autograd.grad(o, (q, k, v), do.cuda().double())


@pytest.mark.parametrize("scale", [1.0, 2.0])   # 2: scores with a standard deviation of 4
@pytest.mark.parametrize("N,D,causal", [(1777, 128, True), (1000, 64, False), (65, 128, False), (129, 64, True)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_ragged_lengths_keep_fp32_accuracy(N, D, causal, dtype, scale):
    """Rounding the result to p bits costs at most 2^-p of a value and about 0.8 * 2^-p of it in the 2-norm; nothing else may show.
    dQ and dK also see delta = rowsum(O dO) of the rounded O, which every kernel of this package forms that way: its rounding error,
    0.8 * 2^-p of sqrt(D) |O| |dO|, stands next to a dP - delta of about the same size, and grows against it as rows become one-hot,
    so they are only looked at for scale 1."""
    q, k, v, do = (draw((1, 2, N, D), 230 + i, dtype) * (scale if i < 2 else 1.0) for i in range(4))
    cos, sin = oracle.precompute_freqs_cis(D, N, 10000.0)
    s = D ** -0.5
    outs = _run(pkg.fused_rope_attention, q, k, v, do, causal, s, cos.cuda(), sin.cuda())
    ulp = 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
    for name, got, ref in zip(("O", "dQ", "dK", "dV"), outs, _exact(q, k, v, do, causal, s, cos, sin)):
        if scale != 1.0 and name in ("dQ", "dK"):
            continue
        err = ((got.double() - ref.cpu()).norm() / ref.cpu().norm()).item()
        assert err < ulp * (1.0 if name in ("O", "dV") else 1.5), (name, err / ulp)


def _exact_grads(q, k, v, do, o, causal, s, cos, sin):
    """dQ, dK, dV in 64 bits with delta = rowsum(O dO) of the given rounded O, as the kernels form it."""
    qd, kd, v, do, o = (t.cuda().double() for t in (q, k, v, do, o))
    half = qd.shape[-1] // 2
    c, sn = cos[:, :half].cuda().double(), sin[:, :half].cuda().double()
    turn = lambda x, w: torch.cat((x[..., :half] * c - w * x[..., half:] * sn, x[..., half:] * c + w * x[..., :half] * sn), -1)   # w = -1: back
    qr, kr = turn(qd, 1.0), turn(kd, 1.0)
    w = qr @ kr.transpose(-1, -2) * s
    if causal:
        w = w.masked_fill(torch.ones_like(w, dtype=torch.bool).triu(1), float("-inf"))
    p = w.softmax(-1)
    ds = p * (do @ v.transpose(-1, -2) - (o * do).sum(-1, keepdim=True)) * s
    return turn(ds @ kr, -1.0), turn(ds.transpose(-1, -2) @ qr, -1.0), p.transpose(-1, -2) @ do


@pytest.mark.parametrize("scale", [1.0, 4.0, 6.0])   # scores with a standard deviation of 1, 16, 36
@pytest.mark.parametrize("N,D,causal", [(1777, 128, True), (1000, 64, False), (1001, 64, True), (65, 128, False)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_ragged_lengths_are_as_accurate_as_fp32_kernels(N, D, causal, dtype, scale):
    """Held against the CUDA-core kernels with fp32 operands (policy 1): the LSE, which is not rounded, by its error, the 16-bit results by
    the share of them that are not the exact result rounded.  Both are proportional to the error before the rounding, and differ
    by what the order of the sums gives (measured: 0.55 to 1.05 of the CUDA-core kernels' share); two 16-bit parts per operand instead of three
    show 5 to 10 times the error."""
    rope = pkg.fused_rope_attn
    q, k, v, do = (draw((1, 4, N, D), 260 + i, dtype) * (scale if i < 2 else 1.0) for i in range(4))
    cos, sin = oracle.precompute_freqs_cis(D, N, 10000.0)
    s = D ** -0.5
    qd, kd, vd, dod, cd, sd = (t.cuda() for t in (q, k, v, do, cos, sin))
    exact_o = _exact(q, k, v, do, causal, s, cos, sin)[0]
    errors = {}
    saved0 = rope._forward(qd, kd, vd, causal, s, cd, sd)
    exact = _exact_grads(q, k, v, do, saved0[3], causal, s, cos, sin)
    half = D // 2
    c, sn = cos[:, :half].cuda().double(), sin[:, :half].cuda().double()
    qr, kr = (torch.cat((x[..., :half] * c - x[..., half:] * sn, x[..., half:] * c + x[..., :half] * sn), -1) for x in (qd.double(), kd.double()))
    w = qr @ kr.transpose(-1, -2) * s
    if causal:
        w = w.masked_fill(torch.ones_like(w, dtype=torch.bool).triu(1), float("-inf"))
    lse = torch.logsumexp(w, -1) / math.log(2.0)
    for policy in (0, 1):
        prev = ext.lib().corope_set_kernel_policy(policy)
        try:
            saved = rope._forward(qd, kd, vd, causal, s, cd, sd)
            grads = rope._backward(*saved0, dod, causal, s)   # both from one O and one LSE
        finally:
            ext.lib().corope_set_kernel_policy(prev)
        ext.check_status()
        errors[policy] = [(saved[4].double() - lse).pow(2).mean().sqrt().item()]
        errors[policy] += [(a != b.to(dtype)).double().mean().item() for a, b in zip((saved[3],) + tuple(grads), (exact_o,) + exact)]
    for name, new, old in zip(("LSE", "O", "dQ", "dK", "dV"), errors[0], errors[1]):
        assert new <= 1.25 * old + (0.0 if name == "LSE" else 1e-4), (name, new, old)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_keys_masked_by_an_infinite_channel(D, dtype):
    # a channel that is 1 in every query and -inf in some keys takes those keys out, as in fp32 arithmetic
    N = 150
    q, k, v = (draw((1, 2, N, D), 290 + i, dtype) for i in range(3))
    q[..., 3] = 1.0
    k[..., 3] = 0.0
    hidden = torch.arange(N) % 3 == 1
    plain = k.clone()
    k[:, :, hidden, 3] = float("-inf")
    o = pkg.flash_attention(q.cuda(), k.cuda(), v.cuda(), False, D ** -0.5)
    ext.check_status()
    seen = [t[:, :, ~hidden] for t in (plain, v)]
    w = q.double() @ seen[0].double().transpose(-1, -2) * D ** -0.5
    ref = w.softmax(-1) @ seen[1].double()
    assert ((o.cpu().double() - ref).norm() / ref.norm()).item() < 2.0 ** (-9 if dtype == torch.bfloat16 else -12)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_ragged_calls_take_the_split_operand_kernels(D, dtype):
    # every check above would pass on the slower CUDA-core kernels too
    B, H, N = 1, 2, 130
    q, k, v, do = (draw((B, H, N, D), 300 + i, dtype) for i in range(4))
    cos, sin = (t.cuda() for t in oracle.precompute_freqs_cis(D, N, 10000.0))
    lib = ext.lib()
    for fn, args in ((pkg.fused_rope_attention, (True, 1.0, cos, sin)), (pkg.fused_rope_attention_theta, (True, 1.0, 1e4)), (pkg.flash_attention, (True, 1.0))):
        _run(fn, q, k, v, do, *args)
        for op in (ext.OP_ROPE_FWD, ext.OP_ROPE_BWD):
            assert (lib.corope_last_kernel_family(op), lib.corope_last_kernel_split(op)) == (0, 1)
    _run(pkg.flash_attention, *(t.float() for t in (q, k, v, do)), True, 1.0)
    for op in (ext.OP_ROPE_FWD, ext.OP_ROPE_BWD):
        assert (lib.corope_last_kernel_family(op), lib.corope_last_kernel_split(op)) == (0, 0)


@pytest.mark.parametrize("N", [1, 31, 33, 65, 97, 130])
@pytest.mark.parametrize("D,causal,dtype", [(128, True, torch.bfloat16), (128, False, torch.bfloat16), (64, True, torch.bfloat16), (128, True, torch.float16)])
def test_plain_attention_at_step_edges(N, D, causal, dtype):
    # 32 streamed rows per warp and step, 64 owned rows; D = 128: two warps share 16 rows and each sees every other 32 streamed ones.  bf16
    # keys are read from the caller's tensor, here a transposed one, f16 keys from their split copies
    B, Hq, Hkv = 2, 6, 2
    q, do = (draw((B, Hq, N, D), 310 + i, dtype) for i in range(2))
    k, v = (draw((B, N, Hkv, D), 312 + i, dtype).transpose(1, 2) for i in range(2))
    outs = _run(pkg.flash_attention, q, k, v, do, causal, D ** -0.5)
    refs = (oracle.attn_gqa_fwd(q, k, v, causal, D ** -0.5),) + tuple(oracle.attn_gqa_bwd(q, k, v, do, causal, D ** -0.5))
    _check(outs, refs, dtype)


@pytest.mark.parametrize("N,D,causal", [(1000, 128, True), (1001, 64, False)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_plain_attention_is_as_accurate_as_fp32_kernels(N, D, causal, dtype):
    q, k, v, do = (draw((1, 4, N, D), 320 + i, dtype) * (2.0 if i < 2 else 1.0) for i in range(4))
    one, zero = torch.ones(N, D), torch.zeros(N, D)
    exact = _exact(q, k, v, do, causal, D ** -0.5, one, zero)
    wrong = {}
    for policy in (0, 1):
        prev = ext.lib().corope_set_kernel_policy(policy)
        try:
            outs = _run(pkg.flash_attention, q, k, v, do, causal, D ** -0.5)
        finally:
            ext.lib().corope_set_kernel_policy(prev)
        wrong[policy] = [(a.to(dtype) != b.cpu().to(dtype)).double().mean().item() for a, b in zip((outs[0], outs[3]), (exact[0], exact[3]))]
    for new, old in zip(*(wrong[x] for x in (0, 1))):   # O, dV
        assert new <= 1.25 * old + 1e-4, wrong
