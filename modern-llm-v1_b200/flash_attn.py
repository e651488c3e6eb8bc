"""Host-side mirror of the reference's flash-attention operator interface.

Same names, argument order and error behaviour as
``modernllm::flash_attn_forward`` / ``flash_attn_backward``
(llm/src/model/flash_attn.h:25-28,47-52; validation llm/src/model/flash_attn.cu:386-407,
433-455) with torch CUDA tensors standing in for ``modernllm::Tensor``:

* caller allocates every input and output, outputs are overwritten in full;
* ``B`` in the two reference-shaped functions is batch x heads (the reference
  kernels know nothing of heads); the ``*_gqa`` variants take (B, T, Hq, Hkv, D)
  and a layout and index the shared KV head directly;
* ``tile_kv`` / ``tile`` are accepted for source compatibility, validated like the
  reference (``<= 0`` raises) and otherwise ignored: tile shapes are compile-time
  properties of the sm_100a kernels;
* bad dtype / device / shape raise ValueError (std::invalid_argument in the
  reference), CUDA failures raise RuntimeError (std::runtime_error).

Tensors are BF16 (the reference's BF16 storage, llm/src/core/dtype.h:34-49), the
logsumexp tensor is FP32.  Everything runs on the current CUDA stream of torch.
There is no CPU or PyTorch fallback.  The argument checks and the call into the C ABI
are native code (csrc/host_binding.cc).
"""
from __future__ import annotations

import torch

from . import _lib

def _dims_ok(B: int, T: int, D: int) -> bool:
    return B > 0 and T > 0 and D > 0


# ----------------------------------------------------------------------------
# GQA-aware entry points (what ModernGPT's attention chain would call)
# ----------------------------------------------------------------------------
def flash_attn_forward_gqa(q, k, v, ctx, L, B, T, Hq, Hkv, D, layout="BHTD", softmax_scale=None):
    """ctx = causal softmax(scale q k^T) v, L = logsumexp rows.  q, ctx: B*Hq*T*D BF16
    elements in `layout`; k, v: B*Hkv*T*D; L: [B, Hq, T] FP32."""
    _lib.host().fwd(q, k, v, ctx, L, B, T, Hq, Hkv, D, layout, softmax_scale)


def flash_attn_backward_gqa(q, k, v, ctx, L, d_ctx, d_q, d_k, d_v, B, T, Hq, Hkv, D, layout="BHTD",
                            softmax_scale=None, mode="auto"):
    """d_q, d_k, d_v (overwritten) for the forward above.  d_k, d_v are Hkv-wide: the
    sum over each group's query heads is done inside the kernel.  mode: "auto", "two_pass" (the
    reference's structure, llm/src/model/flash_attn.cu:475-503, every output bit-reproducible) or
    "one_pass" (D = 64: scores computed once, d_q summed by reduce-adds in no fixed order)."""
    _lib.host().bwd(q, k, v, ctx, L, d_ctx, d_q, d_k, d_v, B, T, Hq, Hkv, D, layout, softmax_scale, mode)


# ----------------------------------------------------------------------------
# Reference-shaped entry points: [B, T, D] with B = batch x heads
# ----------------------------------------------------------------------------
def flash_attn_forward(q, k, v, ctx, L, B, T, D, tile_kv=32):
    """Signature of modernllm::flash_attn_forward (llm/src/model/flash_attn.h:25-28)."""
    if tile_kv <= 0:
        raise ValueError("flash_attn_forward: tile_kv must be > 0")
    if not _dims_ok(B, T, D):
        raise ValueError("flash_attn_forward: shape mismatch (qkv/ctx)")
    flash_attn_forward_gqa(q, k, v, ctx, L, B, T, 1, 1, D, "BHTD")


def flash_attn_backward(q, k, v, ctx, L, d_ctx, d_q, d_k, d_v, B, T, D, tile=16):
    """Signature of modernllm::flash_attn_backward (llm/src/model/flash_attn.h:47-52)."""
    if tile <= 0:
        raise ValueError("flash_attn_backward: tile must be > 0")
    if not _dims_ok(B, T, D):
        raise ValueError("flash_attn_backward: shape mismatch")
    flash_attn_backward_gqa(q, k, v, ctx, L, d_ctx, d_q, d_k, d_v, B, T, 1, 1, D, "BHTD")


# ----------------------------------------------------------------------------
# Decode against a KV cache (the single-token path infer_modern_gpt lacks,
# llm/apps/infer_modern_gpt.cu:253-255)
# ----------------------------------------------------------------------------
def flash_attn_decode(q, kcache, vcache, o, lse, B, L, Hq, Hkv, D, softmax_scale=None, n_splits=0):
    """o[b, h] = softmax(scale q[b, h] . K[b, h/g, :L]) V[b, h/g, :L]; q, o [B, Hq, D] BF16,
    caches [B, Hkv, L, D] BF16, lse [B, Hq] FP32 or None."""
    _lib.host().decode(q, kcache, vcache, o, lse, B, L, Hq, Hkv, D, softmax_scale, n_splits)


def device_status() -> int:
    """Synchronises the current stream and raises RuntimeError if a kernel gave up on a
    bounded wait since the last check; returns 0 otherwise."""
    rc = _lib.load().b200attn_last_device_status(torch.cuda.current_stream().cuda_stream)
    _lib.check(rc, "device_status")
    return rc
