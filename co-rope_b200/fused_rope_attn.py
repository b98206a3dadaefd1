"""Drop-in for the reference's `fused_rope_attn.attention` (fused-rope/fused_rope_attn.py:652-780).

    attention(q, k, v, causal, sm_scale, freqs_cos, freqs_sin, warp_specialize=True) -> o

q, k, v: [B, H, N, D] CUDA tensors of one dtype (bf16, fp16 or fp32).  freqs_cos / freqs_sin: [N, D]
("cat" layout of precompute_freqs_cis) or [N, D/2]; only columns [0, D/2) are read, as in the
reference (fused_rope_attn.py:88-93).
The CUDA kernels are reached through the C ABI in include/corope_b200.h; the checks (those of the reference's entry point,
fused_rope_attn.py:657-661), allocations and autograd nodes are C++ (csrc/torch_binding.cpp).

The kernels take the tensors' own strides, like the reference's (fused_rope_attn.py:709-710): a [B, N, H, D] buffer viewed as
[B, H, N, D] is not copied, and o = empty_like(q) has q's layout (:662).

Device-side errors: kernels never trap; a bounded wait that runs out sets a per-device status word and its pinned host
mirror.  Every call first looks at the mirror (no synchronisation) and raises RuntimeError, clearing the word, if an
earlier call set it; `_ext.check_status()` does the same with a synchronisation.
"""

import torch

try:
    from . import _ext
except ImportError:  # imported as a top-level module (directory on sys.path, the way the reference's scripts import it)
    import _ext

SUPPORTED_HEAD_DIMS = (32, 64, 128)


def _forward(q, k, v, causal, sm_scale, freqs_cos, freqs_sin):
    """Checks + one library call.  Returns what the backward needs: (q, k, v, o, M, cos, sin, table stride)."""
    return _ext.native().rope_forward(q, k, v, causal, sm_scale, freqs_cos, freqs_sin)


def _backward(q, k, v, o, M, cos, sin, tstride, do, causal, sm_scale):
    """One library call on what _forward returned.  Returns (dq, dk, dv)."""
    return _ext.native().rope_backward(q, k, v, o, M, cos, sin, tstride, do, causal, sm_scale)


def attention(q, k, v, causal, sm_scale, freqs_cos, freqs_sin, warp_specialize=True):
    return _ext.native().rope_attention(q, k, v, causal, sm_scale, freqs_cos, freqs_sin)


# ---------------------------------------------------------------------------------------------------------------------
# The same attention with the tables left out of the interface: for callers whose cos / sin tables are the output of the
# reference's precompute_freqs_cis(D, N, theta) (fused-rope/rope_attn_pytorch.py:10-49) the angles can be formed on the
# device from theta, so no [N, D] tables have to exist at all.  The explicit-table entry point above stays the
# general case (other positions, scaled frequencies).
# ---------------------------------------------------------------------------------------------------------------------
def inv_freq_of(theta, D, device):
    """The D/2 frequencies exactly as precompute_freqs_cis computes them (rope_attn_pytorch.py:29), on `device`."""
    return 1.0 / (theta ** (torch.arange(0, D, 2, device=device).float() / D))


def attention_theta(q, k, v, causal, sm_scale, theta):
    """Positions 0 .. N-1, base theta.  O and the gradients are contiguous whatever the inputs' strides are."""
    return _ext.native().theta_attention(q, k, v, causal, sm_scale, theta)
