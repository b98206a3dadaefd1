"""Drop-in for the reference's un-fused flash attention entry point
(fused-rope/flash_attn_v2_triton.py:513-631; the module keeps the reference's name so its scripts can import this one).

    attention(q, k, v, causal, sm_scale, warp_specialize=True) -> o

q: [B, Hq, N, D]; k, v: [B, Hkv, N, D] with Hq % Hkv == 0 -- query head h reads K / V head h // (Hq // Hkv), as the
reference's kernel maps them (:194-196).  No RoPE: callers rotate q / k themselves (the reference's baselines do,
fused-rope/baseline.py).  The backward also takes Hq != Hkv and returns dk / dv summed over each group (the reference's
backward asserts equal strides, i.e. Hq == Hkv, :560); the math is that of assets/flashattn-gqa/attn_gqa_pytorch.py.
The kernels are the fused-RoPE kernels with the rotation switched off, reached through corope_flash_attn_fwd / _bwd of
the C ABI in include/corope_b200.h; checks (as flash_attn_v2_triton.py:517-521), allocations and autograd nodes are C++
(csrc/torch_binding.cpp).  Device-side errors are reported as in fused_rope_attn.py.
"""

try:
    from . import _ext
except ImportError:  # imported as a top-level module (directory on sys.path, the way the reference's scripts import it)
    import _ext

SUPPORTED_HEAD_DIMS = (32, 64, 128)


def attention(q, k, v, causal, sm_scale, warp_specialize=True):
    return _ext.native().flash_attention(q, k, v, causal, sm_scale)
