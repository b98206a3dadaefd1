"""Drop-in for the reference's Co-RoPE GQA entry point
(corope-exp/flash_attn_co_rope_gqa_triton.py:403-580; the module keeps the reference's name so its scripts
can import this one unchanged).

    attention(q, k, v, causal, sm_scale, theta, warp_specialize=False) -> o

q: [B, Hq, N, D]; k, v: [B, Hkv, N, D]; Hq % Hkv == 0 and group size <= 8; causal must be True.
The math is that of corope-exp/corope_attn_gqa_pytorch.py; forward and backward are CUDA kernels reached
through the C ABI in include/corope_b200.h (the reference's backward is dense PyTorch); checks and messages (as
flash_attn_co_rope_gqa_triton.py:407-425), allocations and autograd nodes are C++ (csrc/torch_binding.cpp).

Device-side errors (an expired bounded wait; a gradient term beyond the value range of the 16-bit backward) set a
per-device status word and its pinned host mirror; every call first looks at the mirror and raises RuntimeError if an
earlier call set it (see fused_rope_attn.py).
"""

try:
    from . import _ext
except ImportError:
    import _ext


def _forward(q, k, v, causal, sm_scale, theta):
    """Checks + one library call.  Returns what the backward needs: (q, k, v, o, lse2, a_diag)."""
    return _ext.native().gqa_forward(q, k, v, causal, sm_scale, theta)


def _backward(q, k, v, o, lse2, a_diag, grad_output, sm_scale, theta):
    """One library call on what _forward returned.  Returns (dq, dk, dv); dk / dv are summed over each group."""
    return _ext.native().gqa_backward(q, k, v, o, lse2, a_diag, grad_output, sm_scale, theta)


def attention(q, k, v, causal, sm_scale, theta, warp_specialize=False):
    return _ext.native().gqa_attention(q, k, v, causal, sm_scale, theta)
