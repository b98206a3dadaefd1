"""The fp32 CUDA-core kernels at the edges of their 32- and 64-row tiles, for each head dimension, grouped heads and rows that
cannot be moved in vectors; tolerance: the 1e-4 of the other fp32 tests."""

import ctypes

import pytest
import torch

import oracle
from helpers import draw, ext, maxdiff, pkg

pytestmark = pytest.mark.gpu

TOL_32 = 1e-4


def _run(fn, q, k, v, do, *args):
    qd, kd, vd = (t.requires_grad_(True) for t in (q, k, v))
    o = fn(qd, kd, vd, *args)
    o.backward(do)
    ext.check_status()
    return tuple(t.detach().float().cpu() for t in (o, qd.grad, kd.grad, vd.grad))


@pytest.mark.parametrize("N", [1, 31, 33, 64, 65, 130])
@pytest.mark.parametrize("D,causal", [(32, True), (64, False), (64, True), (128, True), (128, False)])
def test_rope_fp32_at_tile_edges(N, D, causal):
    q, k, v, do = (draw((1, 2, N, D), 400 + i, torch.float32) for i in range(4))
    cos, sin = oracle.precompute_freqs_cis(D, N, 10000.0)
    s = D ** -0.5
    outs = _run(pkg.fused_rope_attention, *(t.cuda() for t in (q, k, v, do)), causal, s, cos.cuda(), sin.cuda())
    refs = (oracle.rope_attn_fwd(q, k, v, causal, s, cos, sin),) + tuple(oracle.rope_attn_bwd(q, k, v, do, causal, s, cos, sin))
    for a, b in zip(outs, refs):
        assert maxdiff(a, b) < TOL_32


@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("D", [32, 64, 128])
def test_grouped_heads_many_ctas_and_unaligned_rows(pad, D):
    # enough 64-row tiles to fill the chip (the 64-row forward CTA), 4 query heads per K / V head, rows of D + pad floats
    B, Hq, Hkv, N = 2, 32, 8, 330
    grid = (ctypes.c_uint32 * 2)()
    assert ext.lib().corope_debug_grid(0, B, Hq, Hkv, N, D, grid) == 0 and list(grid) == [B * Hq, 6]   # 64-row blocks

    def make(heads, seed):
        t = draw((B, heads, N, D), seed, torch.float32)
        buf = torch.zeros((B, heads, N, D + pad), device="cuda")
        buf[..., :D] = t.cuda()
        return t, buf[..., :D]

    (q, qv), (do, dov), (k, kv), (v, vv) = make(Hq, 410), make(Hq, 411), make(Hkv, 412), make(Hkv, 413)
    prev = ext.lib().corope_set_kernel_policy(1)   # aligned rows of D = 64 run on split operands otherwise
    try:
        outs = _run(pkg.flash_attention, qv.detach(), kv.detach(), vv.detach(), dov, True, D ** -0.5)
    finally:
        ext.lib().corope_set_kernel_policy(prev)
    for op in (ext.OP_ROPE_FWD, ext.OP_ROPE_BWD):
        assert (ext.lib().corope_last_kernel_family(op), ext.lib().corope_last_kernel_split(op)) == (0, 0)
    refs = (oracle.attn_gqa_fwd(q, k, v, True, D ** -0.5),) + tuple(oracle.attn_gqa_bwd(q, k, v, do, True, D ** -0.5))
    for a, b in zip(outs, refs):
        assert maxdiff(a, b) < TOL_32


def test_backward_of_a_very_large_group():
    # 32 768 query heads on one K / V head: 65 538 row blocks of one key head.  dK and dV are sums over all of them, so the tolerance is
    # relative to their largest value.
    B, Hq, Hkv, N, D = 1, 32768, 1, 33, 32
    q, do = (draw((B, Hq, N, D), 420 + i, torch.float32) for i in range(2))
    k, v = (draw((B, Hkv, N, D), 422 + i, torch.float32) for i in range(2))
    outs = _run(pkg.flash_attention, *(t.cuda() for t in (q, k, v, do)), True, D ** -0.5)
    refs = (oracle.attn_gqa_fwd(q, k, v, True, D ** -0.5),) + tuple(oracle.attn_gqa_bwd(q, k, v, do, True, D ** -0.5))
    for a, b in zip(outs, refs):
        assert maxdiff(a, b) < TOL_32 * max(1.0, b.abs().max().item())
