"""Per-layer KV cache for token-by-token sampling (csrc/kv_cache.cuh, csrc/attn_decode.cuh).

The reference's sampler keeps no cache: every generated token re-runs the model over the whole
T-token window (llm/apps/infer_modern_gpt.cu:13,253-255), and the cache is listed as future work
(TODO.md, "KV cache for inference").  This class is the attention side of that cache for a
ModernGPT block (llm/src/model/modern_gpt.cu:351-378): per layer a BF16 K and V buffer
[B, Hkv, L_cap, D]; `append` does split_heads + RoPE at the true positions + QK-Norm for the newest
tokens and stores their k and v, `attend` runs attention for them (causal forward over the prompt,
or the split-KV decode kernel for one token), `advance` moves the length once every layer is done.
The B sequences advance in lock step until `set_lengths` gives each its own length (a batch of
prompts of different lengths); from then on `append` and `attend` take one token per sequence at the
sequence's own position.  Like the reference's operators, the caller allocates every
input and output; bad arguments raise ValueError, CUDA failures RuntimeError; there is no CPU or
PyTorch fallback.
"""
from __future__ import annotations

import torch

from . import _lib
from .rope_norm import make_rope_cache


class KVCache:
    def __init__(self, n_layers: int, B: int, Hq: int, Hkv: int, D: int, L_cap: int, device="cuda",
                 rope_base: float = 10000.0, eps: float = 1e-5):
        if min(n_layers, B, Hq, Hkv, D, L_cap) <= 0 or Hq % Hkv != 0:
            raise ValueError("KVCache: sizes must be positive and Hq a multiple of Hkv")
        if D not in (64, 128):
            raise ValueError("KVCache: d_h must be 64 or 128")
        _lib.load()  # fail now, not at the first token, when the CUDA library is missing
        self.n_layers, self.B, self.Hq, self.Hkv, self.D, self.L_cap = n_layers, B, Hq, Hkv, D, L_cap
        self.eps = float(eps)
        self.device = torch.device(device)
        self.k = torch.zeros((n_layers, B, Hkv, L_cap, D), dtype=torch.bfloat16, device=self.device)
        self.v = torch.zeros_like(self.k)
        self.cos, self.sin = make_rope_cache(L_cap, D, rope_base, device=self.device)
        self.length = 0  # tokens held by every layer (the longest sequence's, once lengths differ)
        self.lengths = None  # per-sequence lengths [B] int32 on the device, once set_lengths was called
        self._lens_next = None  # lengths + 1: what the decode kernel reads while the newest token is being attended
        self._lengths_host = None

    def reset(self) -> None:
        """Forgets every token (the buffers keep their bytes; rows >= length are never read)."""
        self.length = 0
        self.lengths = self._lens_next = self._lengths_host = None

    def set_lengths(self, lengths) -> None:
        """Gives every sequence its own length (e.g. after a padded prompt batch went through `append` /
        `attend` / `advance` with the longest prompt's length): rows at and beyond a sequence's length are
        treated as not yet written."""
        host = [int(x) for x in lengths]
        if len(host) != self.B or min(host) < 0 or max(host) > self.L_cap:
            raise ValueError("KVCache.set_lengths: need B lengths in [0, L_cap]")
        self._lengths_host = host
        self.length = max(host)
        self.lengths = torch.tensor(host, dtype=torch.int32, device=self.device)
        self._lens_next = self.lengths + 1

    def append(self, layer: int, xq, xk, xv, gamma_q, gamma_k, q_out) -> None:
        """xq [B, n_new, Hq, D], xk / xv [B, n_new, Hkv, D] (the projection outputs, FP32 or BF16, all the
        same type) are the n_new tokens after the `length` cached ones.  Writes q_out [B, Hq, n_new, D] BF16
        (rotated, normalised, times gamma_q) and the tokens' rows of this layer's K (same chain with gamma_k)
        and V (converted to BF16)."""
        _lib.host().kv_append(self, layer, xq, xk, xv, gamma_q, gamma_k, q_out)

    def attend(self, layer: int, q, ctx, lse, n_new: int = 1, softmax_scale=None) -> None:
        """Attention of the n_new appended tokens over the length + n_new cached ones.  q, ctx: [B, Hq, n_new, D]
        BF16; lse: [B, Hq, n_new] FP32 (may be None for n_new == 1).  n_new == 1 is the split-KV decode kernel;
        n_new > 1 is the causal forward of the new tokens over the cache: a whole prompt into an empty cache, or a
        further chunk of it behind the tokens already cached (chunked prefill; lock-step sequences only)."""
        _lib.host().kv_attend(self, layer, q, ctx, lse, n_new, softmax_scale)

    def advance(self, n_new: int = 1) -> None:
        """Call once per step, after every layer has appended and attended."""
        if n_new <= 0 or self.length + n_new > self.L_cap:
            raise ValueError("KVCache.advance: n_new out of range")
        self.length += n_new
        if self.lengths is not None:
            self._lengths_host = [x + n_new for x in self._lengths_host]
            self.lengths += n_new
            self._lens_next += n_new
