"""Host-side mirror of the fused RoPE + QK-Norm operator (csrc/rope_norm.cuh).

The reference prepares q and k for attention with split_heads -> rope_apply_inplace ->
rmsnorm_forward (llm/src/model/modern_gpt.cu:351-370) and undoes it in the backward with
rmsnorm_backward -> rope_apply_backward_inplace -> merge_heads (llm/src/model/modern_gpt.cu:527-552).
The two functions here do each chain in one pass; argument names follow the reference's operators
(llm/src/model/rope.h, llm/src/model/rmsnorm.h): caller allocates every tensor, outputs are
overwritten, except ``d_gamma``, which is accumulated into as in the reference
(llm/src/model/rmsnorm.h:17).  Bad dtype / device / shape raise ValueError, CUDA failures
RuntimeError.  There is no CPU or PyTorch fallback.
"""
from __future__ import annotations

import ctypes

import numpy as np
import torch

from . import _lib


def make_rope_cache(T_max: int, d_h: int, base: float = 10000.0, device="cuda"):
    """cos, sin tables [T_max, d_h / 2] FP32 with the values of the reference's make_rope_cache
    (llm/src/model/rope.cu:112-128), computed by the library on the host and copied to `device`."""
    if d_h % 2 != 0:
        raise ValueError("d_h must be even")
    cos = np.empty((T_max, d_h // 2), dtype=np.float32)
    sin = np.empty_like(cos)
    lib = _lib.load()
    _lib.check(lib.b200attn_rope_table(T_max, d_h, ctypes.c_float(base), cos.ctypes.data, sin.ctypes.data),
               "make_rope_cache")
    return torch.from_numpy(cos).to(device), torch.from_numpy(sin).to(device)


def rope_qknorm_forward(x, cos, sin, gamma, eps, y, rstd, B, T, H, D, x_layout="BTHD", y_layout="BHTD"):
    """y = RMSNorm(RoPE(x)) * gamma per head row, rstd = 1 / rms (FP32 [B, H, T]).  x: B*T*H rows of D
    elements, BF16 or FP32, in x_layout (BTHD = the projection output where it lies); y: BF16 in y_layout,
    ready for flash_attn_forward_gqa."""
    _lib.host().rope_fwd(x, cos, sin, gamma, eps, y, rstd, B, T, H, D, x_layout, y_layout)


def rope_qknorm_backward(d_y, x, cos, sin, gamma, rstd, d_x, d_gamma, B, T, H, D, x_layout="BTHD", y_layout="BHTD"):
    """d_x (x's type and layout, overwritten) and d_gamma (FP32 [D], accumulated into) from d_y (BF16 in
    y_layout), the forward's input x and its rstd."""
    _lib.host().rope_bwd(d_y, x, cos, sin, gamma, rstd, d_x, d_gamma, B, T, H, D, x_layout, y_layout)


def rope_qknorm_forward_qk(xq, xk, cos, sin, gamma_q, gamma_k, eps, yq, yk, rstd_q, rstd_k, B, T, Hq, Hkv, D,
                           x_layout="BTHD", y_layout="BHTD"):
    """rope_qknorm_forward for q (Hq heads) and k (Hkv heads) in one launch; bit-identical to two calls."""
    _lib.host().rope_fwd_qk(xq, xk, cos, sin, gamma_q, gamma_k, eps, yq, yk, rstd_q, rstd_k, B, T, Hq, Hkv, D, x_layout,
                            y_layout)


def rope_qknorm_backward_qk(d_yq, d_yk, xq, xk, cos, sin, gamma_q, gamma_k, rstd_q, rstd_k, d_xq, d_xk, d_gamma_q,
                            d_gamma_k, B, T, Hq, Hkv, D, x_layout="BTHD", y_layout="BHTD"):
    """rope_qknorm_backward for q and k in one launch; bit-identical to two calls."""
    _lib.host().rope_bwd_qk(d_yq, d_yk, xq, xk, cos, sin, gamma_q, gamma_k, rstd_q, rstd_k, d_xq, d_xk, d_gamma_q, d_gamma_k,
                            B, T, Hq, Hkv, D, x_layout, y_layout)
