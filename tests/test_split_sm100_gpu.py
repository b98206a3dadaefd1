"""The tcgen05 split-operand kernels of ragged lengths where their persistent loops and rings wrap: more items than SMs, sweeps that end
in the middle of a 64-row block, grouped heads whose sweep runs over several query heads, owned blocks that are nearly empty."""

import math

import pytest
import torch

import oracle
from helpers import draw, ext, pkg

pytestmark = pytest.mark.gpu


def _exact(q, k, v, do, causal, s):
    q, k, v, do = (t.cuda().double() for t in (q, k, v, do))
    G = q.shape[1] // k.shape[1]
    ke, ve = (t.repeat_interleave(G, 1) for t in (k, v))
    w = q @ ke.transpose(-1, -2) * s
    if causal:
        w = w.masked_fill(torch.ones(w.shape[-2:], dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    p = w.softmax(-1)
    o = p @ ve
    ds = p * (do @ ve.transpose(-1, -2) - (o * do).sum(-1, keepdim=True)) * s
    fold = lambda t: t.unflatten(1, (k.shape[1], G)).sum(2)
    return o, ds @ ke, fold(ds.transpose(-1, -2) @ q), fold(p.transpose(-1, -2) @ do)


def _run(q, k, v, do, causal, s):
    q, k, v = (t.cuda().requires_grad_(True) for t in (q, k, v))
    o = pkg.flash_attention(q, k, v, causal, s)
    grads = torch.autograd.grad(o, (q, k, v), do.cuda())
    ext.check_status()
    return (o.detach(),) + grads


@pytest.mark.parametrize("B,Hq,Hkv,N", [(2, 40, 40, 257), (1, 160, 160, 65), (1, 12, 3, 385), (3, 8, 1, 191), (1, 2, 2, 1153), (1, 4, 2, 639)])
@pytest.mark.parametrize("D,causal,dtype", [(128, True, torch.bfloat16), (64, False, torch.bfloat16), (64, True, torch.float16), (128, False, torch.float16)])
def test_wraps_of_items_rings_and_sweeps(B, Hq, Hkv, N, D, causal, dtype):
    # one rounding of the result is at most 2^-9 (bf16) or 2^-12 of a value, in the 2-norm about 0.8 of that; dQ and dK also see delta of the
    # rounded O, whose error stands next to a dP - delta of about the same size
    q, do = (draw((B, Hq, N, D), 400 + i, dtype) for i in range(2))
    k, v = (draw((B, Hkv, N, D), 402 + i, dtype) for i in range(2))
    ulp = 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
    for name, got, ref in zip(("O", "dQ", "dK", "dV"), _run(q, k, v, do, causal, D ** -0.5), _exact(q, k, v, do, causal, D ** -0.5)):
        err = ((got.double() - ref).norm() / ref.norm()).item()
        assert err < ulp * (1.0 if name in ("O", "dV") else 1.5), (name, err / ulp)


@pytest.mark.parametrize("D", [64, 128])
def test_results_are_reproducible(D):
    q, do = (draw((1, 12, 700, D), 410 + i, torch.bfloat16) for i in range(2))
    k, v = (draw((1, 4, 700, D), 412 + i, torch.bfloat16) for i in range(2))
    first = _run(q, k, v, do, True, D ** -0.5)
    for _ in range(3):
        assert all(torch.equal(a, b) for a, b in zip(first, _run(q, k, v, do, True, D ** -0.5)))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("N", [40, 150])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gradients_of_keys_masked_by_an_infinite_channel(D, N, dtype):
    # as test_keys_masked_by_an_infinite_channel: hidden keys have no share in O, dK and dV (dQ takes 0 times their -inf)
    q, k, v, do = (draw((1, 2, N, D), 420 + i, dtype) for i in range(4))
    q[..., 3] = 1.0
    k[..., 3] = 0.0
    hidden = torch.arange(N) % 3 == 1
    exact = _exact(q, k[:, :, ~hidden], v[:, :, ~hidden], do, False, D ** -0.5)
    k[:, :, hidden, 3] = float("-inf")
    o, _, dk, dv = _run(q, k, v, do, False, D ** -0.5)
    ulp = 2.0 ** (-9 if dtype == torch.bfloat16 else -12)
    assert ((o.double() - exact[0]).norm() / exact[0].norm()).item() < ulp
    for got, ref, room in ((dk, exact[2], 1.5), (dv, exact[3], 1.0)):
        assert not got[:, :, hidden].any()
        assert ((got[:, :, ~hidden].double() - ref).norm() / ref.norm()).item() < ulp * room


@pytest.mark.parametrize("B,Hq,Hkv,N", [(1, 2, 2, 256), (2, 3, 3, 257), (1, 8, 2, 321), (1, 160, 160, 260), (1, 2, 2, 1024), (1, 3, 1, 703)])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("transposed", [False, True])
def test_fp32_tensors(B, Hq, Hkv, N, causal, transposed):
    # sums of some hundred fp32 terms: 2^-24 of a term and a root of their number; the CUDA-core kernels show 2e-7 to 1.1e-6 here
    def make(H, seed):
        return draw((B, N, H, 64), seed, torch.float32).transpose(1, 2) if transposed else draw((B, H, N, 64), seed, torch.float32)

    q, k, v, do = make(Hq, 440), make(Hkv, 441), make(Hkv, 442), make(Hq, 443)
    lib = ext.lib()
    outs = _run(q, k, v, do, causal, 0.125)
    for op in (ext.OP_ROPE_FWD, ext.OP_ROPE_BWD):
        assert (lib.corope_last_kernel_family(op), lib.corope_last_kernel_split(op)) == (0, 1)
    for name, got, ref in zip(("O", "dQ", "dK", "dV"), outs, _exact(q, k, v, do, causal, 0.125)):
        assert got.dtype == torch.float32 and ((got.double() - ref).norm() / ref.norm()).item() < 1e-6, name


def test_fp32_rows_that_are_not_aligned_stay_on_the_cuda_cores():
    wide = [draw((1, 2, 300, 66), 450 + i, torch.float32) for i in range(4)]
    do = wide[3][..., 1:65]   # rows 4 bytes off
    q, k, v = (w.cuda()[..., 1:65].detach().requires_grad_(True) for w in wide[:3])
    o = pkg.flash_attention(q, k, v, True, 0.125)
    grads = torch.autograd.grad(o, (q, k, v), do.cuda())
    ext.check_status()
    assert ext.lib().corope_last_kernel_split(ext.OP_ROPE_FWD) == 0
    for got, ref in zip((o.detach(),) + grads, _exact(q.detach(), k.detach(), v.detach(), do, True, 0.125)):
        assert ((got.double() - ref).norm() / ref.norm()).item() < 4e-6


def _by_policy(policy, fn):
    prev = ext.lib().corope_set_kernel_policy(policy)
    try:
        return fn()
    finally:
        ext.lib().corope_set_kernel_policy(prev)


def _scaled_channels(N, D, kind, dtype):
    """q, k, v, dO with a rotation pair of channels 1000 times as large as the others, and its partner in the other operand as much smaller,
    so that scores, dP and the gradients of the other channels stay as they are."""
    q, k, v, do = (draw((1, 3, N, D), 460 + i, torch.float32) for i in range(4))
    pairs = lambda c: [c, c + D // 2]
    if kind in ("q", "q and k"):
        q[..., pairs(5)] *= 1000
        k[..., pairs(5)] /= 1000
    if kind in ("k", "q and k"):
        k[..., pairs(9)] *= 1000
        q[..., pairs(9)] /= 1000
    if kind == "v":
        v[..., 7] *= 1000
        do[..., 7] /= 1000
    if kind == "dO":
        do[..., 7] *= 1000
        v[..., 7] /= 1000
    return (t.to(dtype) for t in (q, k, v, do))


@pytest.mark.parametrize("kind", ["q", "k", "q and k", "v", "dO"])
@pytest.mark.parametrize("op,N,causal", [("flash", 512, False), ("rope", 300, True), ("theta", 513, True)])
def test_fp32_channels_of_different_scale(kind, op, N, causal):
    # every channel of every result, held against the CUDA-core kernels (measured: 0.3 to 0.9 of their error; leading parts that share a
    # unit per row had up to 1e-3, 4000 times their error)
    D, s = 64, 0.125
    q, k, v, do = (t.cuda() for t in _scaled_channels(N, D, kind, torch.float32))
    cos, sin = (t.cuda() for t in oracle.precompute_freqs_cis(D, N, 10000.0))
    half = D // 2
    c, sn = (t[:, :half].double() if op != "flash" else torch.full((N, half), x, device="cuda", dtype=torch.float64) for t, x in ((cos, 1.0), (sin, 0.0)))
    turn = lambda x, w: torch.cat((x[..., :half] * c - w * x[..., half:] * sn, x[..., half:] * c + w * x[..., :half] * sn), -1)   # w = -1: back
    o, dq, dk, dv = _exact(turn(q.double(), 1.0), turn(k.double(), 1.0), v, do, causal, s)
    exact = (o, turn(dq, -1.0), turn(dk, -1.0), dv)

    def run():
        x = [t.clone().requires_grad_(True) for t in (q, k, v)]
        out = (pkg.flash_attention(*x, causal, s) if op == "flash" else pkg.fused_rope_attention(*x, causal, s, cos, sin) if op == "rope"
               else pkg.fused_rope_attention_theta(*x, causal, s, 10000.0))
        grads = torch.autograd.grad(out, x, do)
        ext.check_status()
        return (out.detach(),) + grads

    new, old = run(), _by_policy(1, run)
    for name, a, b, ref in zip(("O", "dQ", "dK", "dV"), new, old, exact):
        err_new, err_old = (((t.double() - ref).norm(dim=2) / ref.norm(dim=2)).max().item() for t in (a, b))
        assert err_new <= 1.25 * err_old, (name, err_new, err_old)


@pytest.mark.parametrize("N,D", [(999, 64), (390, 128)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_lse_with_channels_of_different_scale(N, D, dtype):
    # the LSE is not rounded to 16 bits and shows what the score products lose
    q, k, v, _ = (t.cuda() for t in _scaled_channels(N, D, "q and k", dtype))
    one, zero = torch.ones(N, D, device="cuda"), torch.zeros(N, D, device="cuda")
    exact = torch.logsumexp(q.double() @ k.double().transpose(-1, -2) * D ** -0.5, -1) / math.log(2.0)
    run = lambda: (pkg.fused_rope_attn._forward(q, k, v, False, D ** -0.5, one, zero)[4].double() - exact).pow(2).mean().sqrt().item()
    new, old = run(), _by_policy(1, run)
    ext.check_status()
    assert new <= 1.25 * old, (new, old)


@pytest.mark.parametrize("causal", [True, False])
def test_fp32_values_at_the_end_of_the_range(causal):
    # keys hidden by a channel of the lowest finite number, which is no bf16 number, and the largest one in V (where no query sees it alone)
    N, s = 300, 0.125
    q, k, v, do = (draw((1, 2, N, 64), 470 + i, torch.float32) for i in range(4))
    q[..., 3] = 1.0
    k[..., 3] = 0.0
    k[:, :, torch.arange(N) % 3 == 1, 3] = torch.finfo(torch.float32).min
    exact = _exact(q, k, v, do, causal, s)
    for name, got, ref in zip(("O", "dQ", "dK", "dV"), _run(q, k, v, do, causal, s), exact):
        assert ((got.double() - ref).norm() / ref.norm()).item() < 1e-6, name
    v[:, :, 42, 7] = torch.finfo(torch.float32).max
    o, ref = pkg.flash_attention(q.cuda(), k.cuda(), v.cuda(), causal, s).double(), _exact(q, k, v, do, causal, s)[0]
    ext.check_status()
    assert ((o - ref).norm(dim=2) / ref.norm(dim=2)).max().item() < 2e-6   # of every channel


def _same_kinds(outs, refs):
    for name, a, b in zip(("O", "dQ", "dK", "dV"), outs, refs):
        assert torch.equal(a.isnan(), b.isnan()), (name, int(a.isnan().sum()), int(b.isnan().sum()))
        assert torch.equal(a.isinf(), b.isinf()) and torch.equal(a[a.isinf()] > 0, b[b.isinf()] > 0), name


@pytest.mark.parametrize("value", [math.inf, -math.inf, math.nan])
@pytest.mark.parametrize("which", ["v", "do"])
def test_fp32_infinities_in_v_and_do(which, value):
    # infinite or NaN exactly where the CUDA-core kernels are: 0 times an infinity must not come from a part of P that is 0
    t = {n: draw((1, 2, 300, 64), 480 + i, torch.float32) for i, n in enumerate(("q", "k", "v", "do"))}
    t[which][:, 0, 200, 5] = value
    t[which][:, 1, 17, 40] = value
    run = lambda: _run(t["q"], t["k"], t["v"], t["do"], False, 0.125)
    _same_kinds(run(), _by_policy(1, run))


@pytest.mark.parametrize("at", [140, 200, 255, 390])   # in the first and the second 64 columns of a 128-row block, at its end, in the last block
@pytest.mark.parametrize("D,dtype", [(64, torch.float32), (64, torch.bfloat16), (128, torch.bfloat16), (64, torch.float16), (128, torch.float16)])
def test_causal_rows_do_not_see_what_is_not_finite_in_hidden_rows(D, dtype, at):
    # rows in front of a key (behind a query) by its group of 16 rows or more must not change by a bit
    t = [draw((1, h, 400, D), 490 + i, dtype) for i, h in enumerate((4, 2, 2, 4))]
    base = _run(*t, True, D ** -0.5)
    for value in (math.inf, math.nan):
        for which in range(4):
            x = [y.clone() for y in t]
            x[which][:, :, at, 5] = value
            outs = _run(*x, True, D ** -0.5)
            front, behind = slice(0, at // 16 * 16), slice(at // 16 * 16 + 16, None)
            names = ((0, "O", front), (1, "dQ", front)) if which in (1, 2) else ((2, "dK", behind), (3, "dV", behind))
            for i, name, rows in names:
                assert torch.equal(outs[i][:, :, rows], base[i][:, :, rows]), ("QKV"[which:which + 1] or "dO", value, name)


@pytest.mark.parametrize("D,dtype", [(64, torch.float32), (64, torch.float16), (128, torch.bfloat16)])
def test_keys_masked_by_an_infinite_channel_cost_nothing(D, dtype):
    # 0 times an infinity among the smaller products is no reason to form scores one by one (4 to 58 times the time); room for noise
    q, k, v, do = (draw((1, 8, 1000, D), 500 + i, dtype).cuda() for i in range(4))
    q[..., 3] = 1.0
    k[..., 3] = 0.0
    hidden = k.clone()
    hidden[:, :, torch.arange(1000) % 3 == 1, 3] = float("-inf")
    times = {}
    for name, key in (("plain", k), ("hidden", hidden)) * 2:
        x = [t.clone().requires_grad_(True) for t in (q, key, v)]
        spans = []
        for _ in range(8):
            begin, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            begin.record()
            for _ in range(4):
                torch.autograd.grad(pkg.flash_attention(*x, False, D ** -0.5), x, do)
            end.record()
            end.synchronize()
            spans.append(begin.elapsed_time(end))
        times[name] = min(spans)
    ext.check_status()
    assert times["hidden"] < 2.0 * times["plain"], times


@pytest.mark.parametrize("N,D,dtype", [(300, 64, torch.float32), (333, 64, torch.float16), (333, 128, torch.bfloat16)])
def test_tables_that_are_not_aligned(N, D, dtype):
    # rows of the tables 4 bytes off a multiple of 16, an odd number of floats apart: the same bits as from aligned tables
    q, k, v, do = (draw((1, 2, N, D), 510 + i, dtype).cuda() for i in range(4))
    cos, sin = (t[:, :D // 2].cuda() for t in oracle.precompute_freqs_cis(D, N, 10000.0))

    def run(tables):
        x = [t.clone().requires_grad_(True) for t in (q, k, v)]
        o = pkg.fused_rope_attention(*x, True, D ** -0.5, *tables)
        return (o.detach(),) + torch.autograd.grad(o, x, do)

    off = []
    for t in (cos, sin):
        wide = torch.full((N, D // 2 + 3), float("nan"), device="cuda")
        wide[:, 1:D // 2 + 1] = t
        off.append(wide[:, 1:D // 2 + 1])
    for a, b in zip(run((cos.contiguous(), sin.contiguous())), run(off)):
        assert torch.equal(a, b)
    ext.check_status()


def test_without_memory_for_split_copies():
    # a call whose split copies do not fit runs on the CUDA cores, which need none
    H, N, D = 64, 2048, 64
    q, k, v, do = (draw((1, H, N, D), 520 + i, torch.float32).cuda().requires_grad_(i < 3) for i in range(4))
    run = lambda: pkg.flash_attention(q, k, v, True, 0.125)
    with_copies = run()
    assert ext.lib().corope_last_kernel_split(ext.OP_ROPE_FWD) == 1
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    room = q.numel() * 4 + (8 << 20)   # o and the LSE, but not 12 bytes per element of k and v
    try:
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + room) / total)
        o = run()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert ext.lib().corope_last_kernel_split(ext.OP_ROPE_FWD) == 0
    ext.check_status()
    assert ((o - with_copies).norm() / o.norm()).item() < 2e-6


@pytest.mark.parametrize("N,D,dtype", [(400, 64, torch.bfloat16), (333, 128, torch.float16), (300, 64, torch.float32)])
def test_heads_that_share_one_v_through_the_c_abi(N, D, dtype):
    # head strides of 0 in V and dO, which the C entry points take (the Python ones copy such tensors first)
    B, H, L = 1, 3, ext.lib()
    q, k = (draw((B, H, N, D), 530 + i, dtype).cuda() for i in range(2))
    v, do = (draw((B, 1, N, D), 532 + i, dtype).cuda().expand(B, H, N, D) for i in range(2))
    s, code = D ** -0.5, ext.DTYPE_CODES[dtype]
    o, dq, dk, dv = (torch.empty_like(q) for _ in range(4))
    m = torch.empty((B, H, N), device="cuda")
    st = ext.strides_of(q=q, k=k, v=v, o=o, d_o=do, dq=dq, dk=dk, dv=dv)
    assert list(st.v)[1] == 0 and list(st.d_o)[1] == 0
    status, stream = ext.status_word(q.device).data_ptr(), torch.cuda.current_stream().cuda_stream
    ws, n = ext.workspace(ext.OP_FLASH_FWD, B, H, H, N, D, dtype, q.device)
    assert L.corope_flash_attn_fwd_strided(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), m.data_ptr(), B, H, H, N, D, code, 1, s, ws.data_ptr(), n, status,
                                           stream, st) == 0
    ws, n = ext.workspace(ext.OP_FLASH_BWD, B, H, H, N, D, dtype, q.device)
    assert L.corope_flash_attn_bwd_strided(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), do.data_ptr(), m.data_ptr(), dq.data_ptr(), dk.data_ptr(),
                                           dv.data_ptr(), B, H, H, N, D, code, 1, s, ws.data_ptr(), n, status, stream, st) == 0
    ext.check_status()
    tol = 1e-6 if dtype == torch.float32 else 2.0 ** (-9 if dtype == torch.bfloat16 else -12) * 1.5   # as in the tests above
    for name, got, ref in zip(("O", "dQ", "dK", "dV"), (o, dq, dk, dv), _exact(q, k, v, do, True, s)):
        assert ((got.double() - ref).norm() / ref.norm()).item() < tol, name
