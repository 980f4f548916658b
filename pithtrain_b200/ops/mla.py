"""Query / key / value assembly of multi-head latent attention on the kernels of ``csrc/mla.cu`` (math specification:
pithtrain/models/deepseek_v2.py:213-277 of the reference)."""

from __future__ import annotations

from typing import Optional, Tuple

import torch

from .. import _native
from .common import sp, use_native


def _rows(t: torch.Tensor) -> torch.Tensor:
    """2-D with rows readable in 16-byte pieces (a column slice of a wider projection qualifies)."""
    return t if t.stride(1) == 1 and t.stride(0) % 8 == 0 and t.data_ptr() % 16 == 0 else _dense(t)


def _dense(t: torch.Tensor) -> torch.Tensor:
    """Contiguous and 16-byte aligned."""
    t = t.contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


class _SplitColumns(torch.autograd.Function):
    """Contiguous column blocks of a fused projection's output; the gradient is one concatenation (slicing under autograd fills,
    copies and adds one full-width buffer per block)."""

    @staticmethod
    def forward(ctx, x, *sizes):
        ctx.sizes, ctx.shape = sizes, x.shape
        return tuple(t.contiguous() for t in x.split(sizes, dim=-1))

    @staticmethod
    def backward(ctx, *grads):
        like = next(g for g in grads if g is not None)
        lead = ctx.shape[:-1]
        gs = [like.new_zeros((*lead, n)) if g is None else g for g, n in zip(grads, ctx.sizes)]
        return (torch.cat(gs, dim=-1),) + (None,) * len(ctx.sizes)


def split_columns(x: torch.Tensor, sizes) -> Tuple[torch.Tensor, ...]:
    return _SplitColumns.apply(x, *sizes)


class _Assemble(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k_pe, kv, cos, sin, positions, S, H, dn, dr, dv):
        n, dev = q.shape[0], q.device
        q, k_pe, kv = _rows(q), _rows(k_pe), _rows(kv)
        qo, ko = (torch.empty((n, H, dn + dr), dtype=q.dtype, device=dev) for _ in range(2))
        vo = torch.empty((n, H, dv), dtype=q.dtype, device=dev)
        rc = _native.lib().pt_mla_fwd(q.data_ptr(), k_pe.data_ptr(), kv.data_ptr(), q.stride(0), k_pe.stride(0), kv.stride(0), cos.data_ptr(),
                                      sin.data_ptr(), _native.ptr(positions), qo.data_ptr(), ko.data_ptr(), vo.data_ptr(), n, S, H, dn, dr, dv,
                                      cos.shape[0], sp())
        _native.check(rc, "pt_mla_fwd")
        ctx.save_for_backward(cos, sin, positions)
        ctx.cfg = (S, H, dn, dr, dv)
        return qo, ko, vo

    @staticmethod
    def backward(ctx, gq, gk, gv):
        cos, sin, positions = ctx.saved_tensors
        S, H, dn, dr, dv = ctx.cfg
        like = next(g for g in (gq, gk, gv) if g is not None)
        n, dev = like.shape[0], like.device
        full = lambda g, d: like.new_zeros((n, H, d)) if g is None else _dense(g)  # noqa: E731
        gq, gk, gv = full(gq, dn + dr), full(gk, dn + dr), full(gv, dv)
        dq = torch.empty((n, H * (dn + dr)), dtype=like.dtype, device=dev)
        dkpe = torch.empty((n, dr), dtype=like.dtype, device=dev)
        dkv = torch.empty((n, H * (dn + dv)), dtype=like.dtype, device=dev)
        rc = _native.lib().pt_mla_bwd(gq.data_ptr(), gk.data_ptr(), gv.data_ptr(), cos.data_ptr(), sin.data_ptr(), _native.ptr(positions),
                                      dq.data_ptr(), dkpe.data_ptr(), dkv.data_ptr(), n, S, H, dn, dr, dv, cos.shape[0], sp())
        _native.check(rc, "pt_mla_bwd")
        return (dq, dkpe, dkv) + (None,) * 8


def supported(x: torch.Tensor, cos: torch.Tensor, H: int, dn: int, dr: int, dv: int) -> bool:
    """What the kernels take: bf16, 16-byte pieces of every part of a head, the heads' rotary gradients in 48 KB."""
    return (use_native(x) and x.numel() > 0 and cos.dtype == torch.bfloat16 and cos.is_contiguous() and cos.data_ptr() % 16 == 0
            and cos.shape[-1] == dr and dn > 0 and dn % 8 == 0 and dv % 8 == 0 and dr % 16 == 0 and H * dr * 4 <= 48 * 1024)


def mla_assemble(q, k_pe, kv, cos, sin, positions: Optional[torch.Tensor], S: int, H: int, dn: int, dr: int, dv: int):
    """``q [n, H*(dn+dr)]``, ``k_pe [n, dr]``, ``kv [n, H*(dn+dv)]`` -> ``q, k [n,H,dn+dr]``, ``v [n,H,dv]`` with the rotary parts
    rotated (interleaved pairs in, halves out) and the rotary key shared by every head. ``positions`` int32 ``[n]`` or None (row % S)."""
    for t in (k_pe, kv, cos, sin, *(() if positions is None else (positions,))):
        if t.device != q.device:
            raise RuntimeError(f"q on {q.device}, another input on {t.device}")
    n = q.shape[0]
    if not (q.shape == (n, H * (dn + dr)) and k_pe.shape == (n, dr) and kv.shape == (n, H * (dn + dv)) and cos.shape == sin.shape
            and cos.shape[1] == dr and (positions is None or positions.shape == (n,))):
        raise RuntimeError(f"MLA inputs of {H} heads {dn} + {dr} / {dv}: q {tuple(q.shape)}, rotary key {tuple(k_pe.shape)}, kv {tuple(kv.shape)}, "
                           f"tables {tuple(cos.shape)}, {tuple(sin.shape)}, positions {None if positions is None else tuple(positions.shape)}")
    if not q.dtype == k_pe.dtype == kv.dtype == cos.dtype == sin.dtype:
        raise RuntimeError(f"MLA inputs of types {q.dtype}, {k_pe.dtype}, {kv.dtype}, {cos.dtype}, {sin.dtype}")
    pos = None if positions is None else positions.int().contiguous()
    return _Assemble.apply(q, k_pe, kv, cos, _dense(sin), pos, S, H, dn, dr, dv)
