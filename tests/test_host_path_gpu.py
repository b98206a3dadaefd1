"""The C++ host path of the entry points: a device-side failure reaches the host without any call in between, and output
gradients and masks in forms a caller may hand over."""

import threading
import time

import pytest
import torch

import oracle
from helpers import check16, draw, ext, fused_attention, pkg

pytestmark = pytest.mark.gpu


def test_a_failing_kernel_writes_the_host_mirror_itself():
    dev = torch.device("cuda", 0)
    ext.check_status(dev)
    word = ext.status_word(dev)
    assert ext.lib().corope_debug_expire_wait(word.data_ptr(), 100, torch.cuda.current_stream(dev).cuda_stream) == 0
    torch.cuda.synchronize()
    q, k, v = (draw((1, 1, 128, 64), i, torch.bfloat16).cuda() for i in range(3))
    with pytest.raises(RuntimeError, match="0x107e"):
        pkg.flash_attention(q, k, v, True, 0.125)
    pkg.flash_attention(q, k, v, True, 0.125)   # cleared
    ext.check_status(dev)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("backward", [False, True])
def test_a_launch_that_does_not_compute_is_reported(D, backward):
    # the word is set and the mirror clear: what a call on another stream meets after a failure has been raised and before the word has
    # been cleared in stream order.  The kernels skip their work then, so the next call has to raise.
    dev = torch.device("cuda", 0)
    ext.check_status(dev)
    q, k, v, do = (draw((1, 2, 256, D), 10 + i, torch.bfloat16).cuda() for i in range(4))
    cos, sin = (t.cuda() for t in oracle.precompute_freqs_cis(D, 256, 10000.0))
    rope = pkg.fused_rope_attn
    saved = rope._forward(q, k, v, True, D ** -0.5, cos, sin)
    word, mirror = ext.status_word(dev), ext._status(dev).mirror_view
    assert ext.lib().corope_debug_expire_wait(word.data_ptr(), 100, torch.cuda.current_stream(dev).cuda_stream) == 0
    torch.cuda.synchronize()
    mirror[0] = 0
    if backward:
        rope._backward(*saved, do, True, D ** -0.5)
    else:
        rope._forward(q, k, v, True, D ** -0.5, cos, sin)
    torch.cuda.synchronize()
    assert int(word.item()) == 0x107e
    with pytest.raises(RuntimeError, match="0x107e"):
        rope._forward(q, k, v, True, D ** -0.5, cos, sin)
    rope._forward(q, k, v, True, D ** -0.5, cos, sin)   # cleared
    ext.check_status(dev)


def test_broadcast_output_gradient_and_partial_requires_grad():
    # o.sum().backward() hands over a dO with zero strides; only v asks for a gradient
    B, H, N, D = 1, 2, 160, 64
    q, k, v = (draw((B, H, N, D), 300 + i, torch.bfloat16) for i in range(3))
    cos, sin = oracle.precompute_freqs_cis(D, N, 10000.0)
    vd = v.cuda().requires_grad_(True)
    qd = q.cuda()
    fused_attention(qd, k.cuda(), vd, True, D ** -0.5, cos.cuda(), sin.cuda(), False).sum().backward()
    ext.check_status()
    ref = oracle.rope_attn_bwd(q, k, v, torch.ones_like(q), True, D ** -0.5, cos, sin)[2]
    assert qd.grad is None
    # dV of an all-ones gradient is the same for every column: sums of P over the queries, up to ~7 here, each of N terms rounded to bf16
    check16("broadcast dO dV", vd.grad.float().cpu(), ref, 2e-2, torch.bfloat16)


def test_wrong_tables_and_dtypes_raise_the_python_errors():
    q = torch.zeros(1, 1, 128, 64, device="cuda", dtype=torch.bfloat16)
    t = torch.zeros(100, 64, device="cuda")
    with pytest.raises(ValueError, match="cover"):
        fused_attention(q, q, q, True, 1.0, t, t)
    with pytest.raises(AssertionError):
        fused_attention(q, q, q.float(), True, 1.0, t, t)
    with pytest.raises(AssertionError):
        pkg.flash_attention(q, q, q[..., :32], True, 1.0)


@pytest.mark.parametrize("entry", ["rope", "theta", "flash", "corope"])
def test_other_threads_run_while_launches_wait(entry):
    # the GPU is busy for about half a second and the launch queue fills up behind that: the calls block in the launch, and a thread
    # that wants to run every millisecond must not be held up for that time
    q = torch.zeros(1, 1, 128, 64, device="cuda", dtype=torch.bfloat16)
    t = torch.zeros(128, 64, device="cuda")
    call = {"rope": lambda: fused_attention(q, q, q, True, 1.0, t, t), "theta": lambda: pkg.fused_rope_attention_theta(q, q, q, True, 1.0, 1e4),
            "flash": lambda: pkg.flash_attention(q, q, q, True, 1.0), "corope": lambda: pkg.corope_gqa_attention(q, q, q, True, 1.0, 1e4)}[entry]
    call()
    torch.cuda.synchronize()
    stop, longest = threading.Event(), [0.0]

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            longest[0], last = max(longest[0], now - last), now

    thread = threading.Thread(target=tick)
    thread.start()
    try:
        time.sleep(0.01)
        torch.cuda._sleep(10 ** 9)   # cycles: 0.5 s at the highest clock
        began = time.perf_counter()
        for _ in range(4000):
            call()
        took = time.perf_counter() - began
    finally:
        stop.set()
        thread.join()
        torch.cuda.synchronize()
    assert took > 0.3          # the queue did fill up
    assert longest[0] < 0.25, longest   # half of what a held lock shows
