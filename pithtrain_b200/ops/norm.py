"""RMSNorm with an optional fused residual add, forward and backward.

``rmsnorm(x, w, eps)`` returns ``norm(x) * w``; with ``residual`` it returns ``(norm(h) * w, h)``
where ``h = x + residual`` — the pre-norm residual pattern of every decoder layer — in one pass
over memory. ``zero_centered`` uses ``(1 + w)`` as the scale (Qwen3.5,
pithtrain/models/qwen35_moe.py:24-34). The weight gradient is accumulated into the parameter's
gradient buffer directly.
"""

from __future__ import annotations

import torch

from .. import _native
from .common import accumulate_grad


def rmsnorm_ref(x, w, eps, residual=None, zero_centered=False):
    h = x if residual is None else x + residual
    hf = h.float()
    rstd = torch.rsqrt(hf.pow(2).mean(-1, keepdim=True) + eps)
    scale = (1.0 + w.float()) if zero_centered else w.float()
    y = (hf * rstd * scale).to(x.dtype)
    return (y, h) if residual is not None else y


class _RMSNormFn(torch.autograd.Function):
    """On tensor operations: other devices, types and widths than the kernels take."""

    @staticmethod
    def forward(ctx, x, w, eps, residual, zero_centered):
        shape = x.shape
        H = shape[-1]
        x2 = x.reshape(-1, H)
        ctx.has_res = residual is not None
        ctx.zero_centered = zero_centered
        ctx.shape = shape
        h = x2 if residual is None else x2 + residual.reshape(-1, H)
        hf = h.float()
        rstd = torch.rsqrt(hf.pow(2).mean(-1) + eps)
        scale = (1.0 + w.float()) if zero_centered else w.float()
        y = (hf * rstd[:, None] * scale).to(x.dtype)
        ctx.save_for_backward(h, w, rstd)
        ctx.w_ref = w
        if residual is not None:
            return y.view(shape), h.view(shape)
        return y.view(shape)

    @staticmethod
    def backward(ctx, dy, dh=None):
        h, w, rstd = ctx.saved_tensors
        H = h.shape[-1]
        dy2 = dy.reshape(-1, H)
        dh2 = dh.reshape(-1, H) if (ctx.has_res and dh is not None) else None
        hf, g = h.float(), dy2.float()
        xh = hf * rstd[:, None]
        scale = (1.0 + w.float()) if ctx.zero_centered else w.float()
        dw = (g * xh).sum(0)
        gw = g * scale
        dx = rstd[:, None] * (gw - xh * (gw * xh).mean(-1, keepdim=True))
        if dh2 is not None:
            dx = dx + dh2.float()
        dx = dx.to(h.dtype)
        if ctx.needs_input_grad[1]:
            accumulate_grad(ctx.w_ref, dw)
        dx = dx.view(ctx.shape)
        return dx, None, None, (dx if ctx.has_res else None), None


def rmsnorm(x, w, eps=1e-6, residual=None, zero_centered=False):
    if (x.is_cuda and x.dtype is torch.bfloat16 and w.dtype is torch.bfloat16 and x.shape[-1] % 8 == 0 and x.shape[-1] <= 8192
            and (residual is None or residual.dtype is torch.bfloat16)):
        return _native.host().rmsnorm(x, w, eps, residual, zero_centered)
    return _RMSNormFn.apply(x, w, eps, residual, zero_centered)


class RMSNorm(torch.nn.Module):
    def __init__(self, dim: int, eps: float = 1e-6, zero_centered: bool = False, device=None, dtype=None):
        super().__init__()
        self.eps = eps
        self.zero_centered = zero_centered
        init = torch.zeros if zero_centered else torch.ones
        self.weight = torch.nn.Parameter(init(dim, device=device, dtype=dtype))
        self.weight._init_fill = 0.0 if zero_centered else 1.0

    def forward(self, x, residual=None):
        return rmsnorm(x, self.weight, self.eps, residual, self.zero_centered)
