"""The passes around an attention whose q projection also emits a per-head output gate, on the kernels of ``csrc/gated_attn.cu``:
zero-centred per-head RMSNorm and partial rotate-half RoPE of q and k on the packed projection, and the sigmoid gate of the
output (math specification: pithtrain/models/qwen35_moe.py of the reference). Norm weight gradients are accumulated into the
parameters' gradient buffers."""

from __future__ import annotations

import torch

from .. import _native
from .common import accumulate_colsum, accumulate_colsum_pair, sp, use_native


def _dense(t: torch.Tensor) -> torch.Tensor:
    """Contiguous and 16-byte aligned."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def gated_attn_supported(qkv: torch.Tensor, q_w: torch.Tensor, k_w: torch.Tensor, rope_dim: int, Hq: int, Hkv: int, D: int) -> bool:
    """bf16, heads of 64, 128 or 256 channels (8 to a lane) and a rotation of a multiple of 16 of them (a partner in another lane)."""
    return (use_native(qkv) and D in (64, 128, 256) and 0 < rope_dim <= D and rope_dim % 16 == 0 and qkv.dim() == 2 and qkv.shape[0] > 0
            and qkv.shape[1] == 2 * (Hq + Hkv) * D
            and all(w.dtype == torch.bfloat16 and w.device == qkv.device and w.shape == (D,) and w.is_contiguous() and w.data_ptr() % 16 == 0
                    for w in (q_w, k_w)))


class _Pre(torch.autograd.Function):
    @staticmethod
    def forward(ctx, qkv, q_w, k_w, cos, sin, Hq, Hkv, D, eps):
        qkv, cos, sin = _dense(qkv), _dense(cos), _dense(sin)
        n = qkv.shape[0]
        q, k, v = (torch.empty((n, h, D), dtype=qkv.dtype, device=qkv.device) for h in (Hq, Hkv, Hkv))
        rstd = torch.empty((n, Hq + Hkv), dtype=torch.float32, device=qkv.device)
        rc = _native.lib().pt_gated_attn_pre_fwd(qkv.data_ptr(), q_w.data_ptr(), k_w.data_ptr(), cos.data_ptr(), sin.data_ptr(), q.data_ptr(),
                                                 k.data_ptr(), v.data_ptr(), rstd.data_ptr(), n, Hq, Hkv, D, cos.shape[1], qkv.stride(0),
                                                 float(eps), sp())
        _native.check(rc, "pt_gated_attn_pre_fwd")
        ctx.save_for_backward(qkv, q_w, k_w, cos, sin, rstd)
        ctx.heads, ctx.refs = (Hq, Hkv, D), (q_w, k_w)
        return q, k, v, qkv[:, :2 * Hq * D].view(n, Hq, 2, D)[:, :, 1]

    @staticmethod
    def backward(ctx, dq, dk, dv, dgate):
        qkv, q_w, k_w, cos, sin, rstd = ctx.saved_tensors
        Hq, Hkv, D = ctx.heads
        n = qkv.shape[0]
        dq, dk, dv, dgate = (torch.zeros((n, h, D), dtype=qkv.dtype, device=qkv.device) if t is None else _dense(t)
                             for t, h in ((dq, Hq), (dk, Hkv), (dv, Hkv), (dgate, Hq)))
        L = _native.lib()
        dqkv = torch.empty_like(qkv)
        part = torch.empty((L.pt_gated_attn_parts(n, Hq, Hkv, D), 2 * D), dtype=torch.float32, device=qkv.device)
        rc = L.pt_gated_attn_pre_bwd(dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), dgate.data_ptr(), qkv.data_ptr(), q_w.data_ptr(), k_w.data_ptr(),
                                     cos.data_ptr(), sin.data_ptr(), rstd.data_ptr(), dqkv.data_ptr(), part.data_ptr(), n, Hq, Hkv, D,
                                     cos.shape[1], qkv.stride(0), sp())
        _native.check(rc, "pt_gated_attn_pre_bwd")
        if all(ctx.needs_input_grad[1:3]):
            accumulate_colsum_pair(*ctx.refs, part, D)
        else:
            for i, ref in enumerate(ctx.refs):
                if ctx.needs_input_grad[1 + i]:
                    accumulate_colsum(ref, part, i * D, (i + 1) * D)
        return (dqkv,) + (None,) * 8


def gated_attn_pre(qkv, q_w, k_w, cos, sin, Hq: int, Hkv: int, D: int, eps: float):
    """``qkv [n, 2*(Hq+Hkv)*D]`` (q and gate interleaved per head, then k, then v), ``cos``/``sin [n, R]`` ->
    ``q [n,Hq,D], k [n,Hkv,D], v [n,Hkv,D]`` and the gate ``[n,Hq,D]``, a view of the packed rows."""
    if not cos.device == sin.device == qkv.device:
        raise RuntimeError(f"qkv on {qkv.device}, rotary tables on {cos.device} and {sin.device}")
    if not (cos.shape == sin.shape and cos.shape[0] == qkv.shape[0] and cos.dtype == sin.dtype == qkv.dtype):
        raise RuntimeError(f"rotary rows {tuple(cos.shape)}, {tuple(sin.shape)} of {cos.dtype}, {sin.dtype} for qkv {tuple(qkv.shape)} of {qkv.dtype}")
    return _Pre.apply(qkv, q_w, k_w, cos, sin, Hq, Hkv, D, eps)


class _Post(torch.autograd.Function):
    @staticmethod
    def forward(ctx, o, gate):
        o = _dense(o)
        n, H, D = o.shape
        y = torch.empty_like(o)
        rc = _native.lib().pt_gated_attn_post_fwd(o.data_ptr(), gate.data_ptr(), gate.stride(0), y.data_ptr(), n, H, D, sp())
        _native.check(rc, "pt_gated_attn_post_fwd")
        ctx.save_for_backward(o, gate)
        return y

    @staticmethod
    def backward(ctx, dy):
        o, gate = ctx.saved_tensors
        dy = _dense(dy)
        n, H, D = o.shape
        d_o, dgate = torch.empty_like(o), torch.empty_like(o)
        rc = _native.lib().pt_gated_attn_post_bwd(dy.data_ptr(), o.data_ptr(), gate.data_ptr(), gate.stride(0), d_o.data_ptr(), dgate.data_ptr(),
                                                  n, H, D, sp())
        _native.check(rc, "pt_gated_attn_post_bwd")
        return d_o, dgate


def gated_attn_post(o, gate):
    """``o [n,H,D] * sigmoid(gate)``; ``gate`` is the view that :func:`gated_attn_pre` returned."""
    if gate.shape != o.shape:
        raise RuntimeError(f"gate {tuple(gate.shape)} for an output {tuple(o.shape)}")
    return _Post.apply(o, gate)
