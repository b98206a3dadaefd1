"""Co-RoPE outside the whole tiles of its mma kernels -- D = 64, ragged lengths, fp32 tensors -- at the edges of the 8-row CTAs and
of the 32- and 64-key tiles, for every kind of group size; and the accuracy of the 16-bit results: rounding, nothing else."""

import os

import pytest
import torch

import oracle
from helpers import check16, corope_attention, draw, ext, maxdiff, run_corope

pytestmark = pytest.mark.gpu

TOL_32, TOL_FWD_16, TOL_BWD_16 = 1e-4, 1e-2, 2e-2


def _label():
    return os.environ.get("PYTEST_CURRENT_TEST", "?").split("::")[-1].split(" ")[0]


def _case(B, Hq, Hkv, N, D, dtype, seed):
    return tuple(draw((B, h, N, D), seed + x, dtype) for x, h in enumerate((Hq, Hkv, Hkv, Hq)))


@pytest.mark.parametrize("N", [1, 9, 31, 33, 63, 65, 130])
@pytest.mark.parametrize("D,Hq,Hkv", [(64, 4, 1), (128, 6, 2), (64, 8, 1), (128, 2, 2)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_16_bit_edges(N, D, Hq, Hkv, dtype):
    q, k, v, do = _case(1, Hq, Hkv, N, D, dtype, 500)
    outs = run_corope(q, k, v, do, D ** -0.5, 10000.0)
    check16(_label() + " O", outs[0], oracle.corope_gqa_fwd(q, k, v, True, D ** -0.5, 10000.0), TOL_FWD_16, dtype, strict=True)
    for name, got, ref in zip("qkv", outs[1:], oracle.corope_gqa_bwd(q, k, v, do, True, D ** -0.5, 10000.0)):
        check16(_label() + " d" + name, got, ref, TOL_BWD_16, dtype)


@pytest.mark.parametrize("N", [1, 9, 33, 65])
@pytest.mark.parametrize("D,Hq,Hkv", [(32, 4, 1), (64, 3, 1), (64, 8, 1), (128, 4, 2), (128, 8, 1), (128, 5, 1)])
def test_fp32_edges(N, D, Hq, Hkv):
    q, k, v, do = _case(2, Hq, Hkv, N, D, torch.float32, 520)
    outs = run_corope(q, k, v, do, D ** -0.5, 10000.0)
    refs = (oracle.corope_gqa_fwd(q, k, v, True, D ** -0.5, 10000.0),) + tuple(oracle.corope_gqa_bwd(q, k, v, do, True, D ** -0.5, 10000.0))
    for x, (a, b) in enumerate(zip(outs, refs)):   # tolerances of the other fp32 Co-RoPE tests
        assert maxdiff(a, b) < (TOL_32 if x == 0 else 2 * TOL_32)


def _exact_o(q, k, v, s, theta):
    """O in 64 bits."""
    q, k, v = (t.double() for t in (q, k, v))
    (B, Hq, N, D), Hkv = q.shape, k.shape[1]
    G, half = Hq // Hkv, D // 2
    w = theta ** (-torch.arange(0, D, 2, dtype=torch.float64, device=q.device) / D)
    hidden = torch.ones(N, N, dtype=torch.bool, device=q.device).triu(1)
    o = torch.empty_like(q)
    for b in range(B):
        for g in range(Hkv):
            z = torch.sigmoid(q[b, g * G] @ k[b, g].T * s).masked_fill(hidden, 0.0)
            a = z.cumsum(1)
            delta = a.diagonal()[:, None] - a
            score = 0
            for p in range(half):
                c, sn = torch.cos(delta * w[p]), torch.sin(delta * w[p])
                k1, k2 = k[b, g, :, p], k[b, g, :, p + half]
                score = score + q[b, g * G:(g + 1) * G, :, p, None] * (k1 * c + k2 * sn) + q[b, g * G:(g + 1) * G, :, p + half, None] * (k2 * c - k1 * sn)
            o[b, g * G:(g + 1) * G] = (score * s).masked_fill(hidden, float("-inf")).softmax(-1) @ v[b, g]
    return o


@pytest.mark.parametrize("N,D", [(500, 128), (333, 64), (512, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_16_bit_results_are_rounded_only(N, D, dtype):
    """Rounding to p bits costs about 0.8 * 2^-p of a value in the 2-norm; nothing else may show."""
    q, k, v, do = _case(1, 8, 2, N, D, dtype, 540)
    o = run_corope(q, k, v, do, D ** -0.5, 10000.0)[0]
    ref = _exact_o(q.cuda(), k.cuda(), v.cuda(), D ** -0.5, 10000.0).cpu()
    ulp = 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
    assert ((o.double() - ref).norm() / ref.norm()).item() < ulp


@pytest.mark.parametrize("scale", [1.0, 0.3, 2.0])
@pytest.mark.parametrize("N,D", [(333, 64), (700, 128), (512, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_16_bit_results_are_as_accurate_as_fp32_kernels(N, D, dtype, scale):
    """The share of results that are not the exact result rounded is proportional to the error before the rounding: held against the
    CUDA-core kernel with fp32 operands (policy 1).  Two bf16 parts per operand, or f16 probabilities that sink into the subnormals,
    show 2 to 10 times that share at scale 0.3, where the phases leave the least error of their own."""
    q, k, v, _ = _case(1, 8, 2, N, D, torch.float32, 560)
    q, k, v = (q * scale).to(dtype), (k * scale).to(dtype), v.to(dtype)
    ref = _exact_o(q.cuda(), k.cuda(), v.cuda(), D ** -0.5, 10000.0).to(dtype)
    wrong = {}
    for policy in (0, 1):
        prev = ext.lib().corope_set_kernel_policy(policy)
        try:
            o = corope_attention(q.cuda(), k.cuda(), v.cuda(), True, D ** -0.5, 10000.0)
        finally:
            ext.lib().corope_set_kernel_policy(prev)
        ext.check_status()
        wrong[policy] = (o != ref).double().mean().item()
    assert wrong[0] <= 1.15 * wrong[1] + 1e-4, wrong


@pytest.mark.parametrize("D", [64, 128])
def test_f16_keys_of_any_magnitude(D):
    # rows of K from the subnormals to the largest f16 numbers, one of zeros, with a query that makes scores of order one of them
    N, dtype = 100, torch.float16
    q, k, v, _ = _case(1, 4, 1, N, D, torch.float32, 580)
    k = k * torch.logspace(-7, 4, N).view(1, 1, N, 1)
    k[:, :, 7] = 0
    k = k.clamp(-65504, 65504).to(dtype)
    q, v = q.to(dtype), v.to(dtype)
    for s in (1e-3, 1e-5):
        o = run_corope(q, k, v, None, s, 10000.0)[0]
        ref = _exact_o(q.cuda(), k.cuda(), v.cuda(), s, 10000.0).cpu()
        assert ((o.double() - ref).norm() / ref.norm()).item() < 2.0 ** -12   # the rounding of O


def test_unaligned_f16_rows_at_a_whole_tile_length():
    # N and D of the mma kernels, rows that they cannot read: the split-operand kernel with its row factors in the workspace
    B, Hq, Hkv, N, D, dtype = 1, 8, 2, 192, 128, torch.float16
    q, k, v, _ = _case(B, Hq, Hkv, N, D, dtype, 590)
    padded = [torch.zeros(t.shape[:3] + (D + 2,), dtype=dtype, device="cuda") for t in (q, k, v)]
    for buf, t in zip(padded, (q, k, v)):
        buf[..., :D] = t.cuda()
    o = corope_attention(*(b[..., :D] for b in padded), True, D ** -0.5, 10000.0)
    ext.check_status()
    assert ext.lib().corope_last_kernel_split(ext.OP_GQA_FWD) == 1
    ref = _exact_o(q.cuda(), k.cuda(), v.cuda(), D ** -0.5, 10000.0)
    assert ((o.double() - ref).norm() / ref.norm()).item() < 2.0 ** -12


@pytest.mark.parametrize("N,D", [(130, 128), (128, 64), (130, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_16_bit_forwards_outside_whole_tiles_take_the_split_operand_kernel(N, D, dtype):
    q, k, v, _ = _case(1, 4, 2, N, D, dtype, 600)
    run_corope(q, k, v, None, D ** -0.5, 10000.0)
    assert (ext.lib().corope_last_kernel_family(ext.OP_GQA_FWD), ext.lib().corope_last_kernel_split(ext.OP_GQA_FWD)) == (0, 1)
    run_corope(q.float(), k.float(), v.float(), None, D ** -0.5, 10000.0)
    assert ext.lib().corope_last_kernel_split(ext.OP_GQA_FWD) == 0
