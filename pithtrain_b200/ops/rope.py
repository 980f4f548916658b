"""Rotary embeddings and the fused per-head QK-RMSNorm + RoPE on the packed QKV projection.

``qk_norm_rope(qkv, q_w, k_w, cos, sin, ...)`` takes the output of the fused q/k/v GEMM
``[tokens, (Hq + 2*Hkv) * D]`` and returns ``q[tokens,Hq,D]``, ``k[tokens,Hkv,D]`` (normalised when
weights are given, rotated by rotate-half RoPE) and ``v`` as a strided view of the input — one
kernel instead of the norm / mul / cat / rotate chain of pithtrain/models/qwen3_moe.py:140-168.
``cos``/``sin`` are ``[max_pos, D]`` tables (bf16 in the reference); ``positions`` optionally gives
each token's position (packed sequences, zigzag context parallelism).
"""

from __future__ import annotations

from typing import Optional

import torch

from .. import _native
from .common import use_native


def rotate_half(x):
    h = x.shape[-1] // 2
    return torch.cat((-x[..., h:], x[..., :h]), dim=-1)


def apply_rope_ref(x, cos, sin):
    """x [..., tokens, heads, D]; cos/sin [tokens, D]."""
    return x * cos.unsqueeze(-2) + rotate_half(x) * sin.unsqueeze(-2)


def _head_norm_ref(x, w, eps, zero_centered):
    xf = x.float()
    y = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps)
    scale = (1.0 + w.float()) if zero_centered else w.float()
    return (y * scale).to(x.dtype)


def qk_norm_rope_ref(qkv, q_w, k_w, cos, sin, Hq, Hkv, D, eps, positions=None, S=None, zero_centered=False):
    n = qkv.shape[0]
    q = qkv[:, : Hq * D].reshape(n, Hq, D)
    k = qkv[:, Hq * D:(Hq + Hkv) * D].reshape(n, Hkv, D)
    v = qkv[:, (Hq + Hkv) * D:].reshape(n, Hkv, D)
    if q_w is not None:
        q = _head_norm_ref(q, q_w, eps, zero_centered)
        k = _head_norm_ref(k, k_w, eps, zero_centered)
    if positions is None:
        positions = torch.arange(n, device=qkv.device) % S
    c, s = cos[positions.long()].to(q.dtype), sin[positions.long()].to(q.dtype)
    return apply_rope_ref(q, c, s), apply_rope_ref(k, c, s), v


def qk_norm_rope(qkv: torch.Tensor, q_w: Optional[torch.Tensor], k_w: Optional[torch.Tensor],
                 cos: torch.Tensor, sin: torch.Tensor, Hq: int, Hkv: int, D: int, eps: float = 1e-6,
                 positions: Optional[torch.Tensor] = None, S: Optional[int] = None, zero_centered: bool = False):
    """Returns ``(q[n,Hq,D], k[n,Hkv,D], v[n,Hkv,D])`` from packed ``qkv[n, (Hq+2Hkv)*D]``."""
    if S is None:
        S = qkv.shape[0]
    if (use_native(qkv) and D in (64, 128) and cos.dtype == torch.bfloat16 and cos.shape[-1] == D
            and qkv.stride(1) == 1 and (q_w is None or q_w.dtype == torch.bfloat16)):
        return _native.host().qk_norm_rope(qkv, q_w, k_w, cos, sin, positions, Hq, Hkv, D, eps, S, zero_centered)
    return qk_norm_rope_ref(qkv, q_w, k_w, cos, sin, Hq, Hkv, D, eps, positions, S, zero_centered)
