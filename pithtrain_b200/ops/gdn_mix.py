"""The elementwise passes of a Gated DeltaNet layer on the kernels of ``csrc/gdn_mix.cu``: the causal depthwise convolution
with its SiLU, the l2 norm of q and k and their repetition over the value heads, and the gated RMSNorm of the output
(math specification: pithtrain/models/qwen35_moe.py:40-47,67-113 of the reference). Weight gradients are accumulated into the
parameters' gradient buffers."""

from __future__ import annotations

import torch

from .. import _native
from .common import accumulate_colsum, sp, use_native


def _dense(t: torch.Tensor) -> torch.Tensor:
    """Contiguous and 16-byte aligned."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def conv_supported(x: torch.Tensor, weight: torch.Tensor, nk: int, nv: int, dk: int, dv: int) -> bool:
    """Heads of 128 channels, four taps, bf16: what a warp of the kernels holds in registers."""
    return (use_native(x) and weight.device == x.device and weight.dtype == torch.bfloat16 and weight.is_contiguous() and weight.data_ptr() % 16 == 0 and dk == 128
            and dv == 128 and nv % nk == 0 and weight.shape == ((2 * nk + nv) * 128, 1, 4) and x.dim() == 3 and x.shape[2] == weight.shape[0]
            and 0 < x.shape[0] <= 65535 and 0 < x.shape[1] <= 65535 * 32)


class _ConvQKV(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, nk, nv):
        x = _dense(x)
        B, S, _ = x.shape
        q, k, v = (torch.empty((B, S, nv, 128), dtype=x.dtype, device=x.device) for _ in range(3))
        rc = _native.lib().pt_gdn_conv_fwd(x.data_ptr(), weight.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), B, S, nk, nv, sp())
        _native.check(rc, "pt_gdn_conv_fwd")
        ctx.save_for_backward(x, weight)
        ctx.heads, ctx.w_ref = (nk, nv), weight
        return q, k, v

    @staticmethod
    def backward(ctx, dq, dk, dv):
        x, weight = ctx.saved_tensors
        nk, nv = ctx.heads
        B, S, C = x.shape
        dq, dk, dv = ((torch.zeros((B, S, nv, 128), dtype=x.dtype, device=x.device) if t is None else _dense(t)) for t in (dq, dk, dv))
        L = _native.lib()
        dx = torch.empty_like(x)
        part = torch.empty((L.pt_gdn_conv_parts(B, S), C * 4), dtype=torch.float32, device=x.device)
        rc = L.pt_gdn_conv_bwd(x.data_ptr(), weight.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), dx.data_ptr(), part.data_ptr(),
                               B, S, nk, nv, sp())
        _native.check(rc, "pt_gdn_conv_bwd")
        if ctx.needs_input_grad[1]:
            accumulate_colsum(ctx.w_ref, part)
        return dx, None, None, None


def conv_qkv(x: torch.Tensor, weight: torch.Tensor, nk: int, nv: int):
    """``x [B,S,(2nk+nv)*128]`` -> ``q, k, v [B,S,nv,128]``: SiLU of the causal convolution with ``weight [C,1,4]``, q and k
    heads normalised to length 1 and repeated ``nv / nk`` times."""
    return _ConvQKV.apply(x, weight, nk, nv)


class _GatedNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, z, weight, eps):
        x, z = _dense(x), _dense(z)
        out = torch.empty_like(x)
        rc = _native.lib().pt_gdn_gnorm_fwd(x.data_ptr(), z.data_ptr(), weight.data_ptr(), out.data_ptr(), x.shape[0], float(eps), sp())
        _native.check(rc, "pt_gdn_gnorm_fwd")
        ctx.save_for_backward(x, z, weight)
        ctx.eps, ctx.w_ref = float(eps), weight
        return out

    @staticmethod
    def backward(ctx, d):
        x, z, weight = ctx.saved_tensors
        d = _dense(d)
        L = _native.lib()
        dx, dz = torch.empty_like(x), torch.empty_like(x)
        part = torch.empty((L.pt_gdn_gnorm_parts(x.shape[0]), 128), dtype=torch.float32, device=x.device)
        rc = L.pt_gdn_gnorm_bwd(d.data_ptr(), x.data_ptr(), z.data_ptr(), weight.data_ptr(), dx.data_ptr(), dz.data_ptr(), part.data_ptr(),
                                x.shape[0], ctx.eps, sp())
        _native.check(rc, "pt_gdn_gnorm_bwd")
        if ctx.needs_input_grad[2]:
            accumulate_colsum(ctx.w_ref, part)
        return dx, dz, None, None


def gated_norm_supported(x: torch.Tensor, z: torch.Tensor, weight: torch.Tensor) -> bool:
    return (use_native(x) and z.device == weight.device == x.device and _native.on_current_device(x)
            and z.dtype == weight.dtype == torch.bfloat16 and x.dim() == 2 and x.shape[1] == 128 and z.shape == x.shape
            and x.shape[0] > 0 and weight.shape == (128,) and weight.is_contiguous() and weight.data_ptr() % 16 == 0)


def gated_norm(x: torch.Tensor, z: torch.Tensor, weight: torch.Tensor, eps: float) -> torch.Tensor:
    """``rmsnorm(x) * weight * silu(z)`` over rows of 128."""
    return _GatedNorm.apply(x, z, weight, eps)
