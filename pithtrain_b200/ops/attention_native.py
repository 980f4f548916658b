"""The framework's own attention kernels (``csrc/attention.cu`` forward, ``csrc/attention_bwd.cu`` and
``csrc/attention_bwd_split.cu`` backward).

tcgen05 / TMEM / TMA kernels for bf16 attention in the token-major ``[B, S, H, D]`` layout the projections write:
causal or unmasked, GQA, sliding windows, packed documents (``cu_seqlens``), learned per-head sinks, and the head
dims of the four model families (64, 128, 192/128 for MLA, 256). They take the role of the reference's
FlashAttention-4 wrapper (pithtrain/operators/flash_attn_v4.py:17-99). ``ops.attention.attention`` calls
:func:`supported` and then :func:`attention`; shapes outside the kernels' range (fp32 inputs, other head dims,
CPU tensors) use the fp32 math of ``ops.attention.attention_ref``.

Windows and documents reach the kernels as one int32 vector ``row_lo[B*Sq]``: the first key each query row may see.
A key ``kp`` is visible to the query at absolute position ``qpos`` iff ``row_lo <= kp <= qpos`` (causal) or
``row_lo <= kp < Sk`` (unmasked).
"""

from __future__ import annotations

from typing import Optional, Tuple

import torch

ENABLED = True
_DIMS = {(64, 64), (128, 128), (192, 128), (256, 256)}
_BWD_DIMS = {(64, 64), (128, 128)}  # of csrc/attention_bwd.cu, for lengths that are a multiple of 4 (why: csrc/host_ops.cpp)
_ROW_LO_CACHE: dict = {}


def _token_major(t: torch.Tensor) -> bool:
    """``[B, S, H, D]`` whose (H, D) block is contiguous and whose tokens are equally spaced, so that the tensor is a
    2-D ``[B*S, H*D]`` matrix with one row pitch (a slice of a fused qkv projection output qualifies)."""
    B, S, H, D = t.shape
    sb, ss, sh, sd = t.stride()
    return sd == 1 and (H == 1 or sh == D) and (B == 1 or sb == S * ss) and ss % 8 == 0 and t.data_ptr() % 16 == 0


def supported(q, k, v, causal, window_left, sinks, cu_seqlens) -> bool:
    if not (ENABLED and q.is_cuda and q.dim() == 4):
        return False
    if q.dtype != torch.bfloat16 or k.dtype != torch.bfloat16 or v.dtype != torch.bfloat16:
        return False
    if (q.shape[-1], v.shape[-1]) not in _DIMS or k.shape[-1] != q.shape[-1]:
        return False
    if k.shape[2] != v.shape[2] or q.shape[2] % k.shape[2] != 0 or k.shape[1] != v.shape[1]:
        return False
    if cu_seqlens is not None and (q.shape[0] != 1 or q.shape[1] != k.shape[1]):
        return False
    return True


def row_lower_bounds(B: int, Sq: int, q_off: int, window_left: Optional[int], cu_seqlens: Optional[torch.Tensor],
                     device) -> Optional[torch.Tensor]:
    """int32 ``[B*Sq]``: first visible key of each query row, or None when every row starts at key 0."""
    has_w = window_left is not None and window_left >= 0
    if not has_w and cu_seqlens is None:
        return None
    from .. import _native

    if (cu_seqlens is not None and _native.on_current_device(cu_seqlens) and cu_seqlens.dim() == 1 and cu_seqlens.numel() >= 2
            and B * Sq > 0 and cu_seqlens.device == torch.device(device)):
        cu = cu_seqlens.to(torch.int32).contiguous()
        lo = torch.empty(B * Sq, dtype=torch.int32, device=device)
        rc = _native.lib().pt_row_lower_bounds(cu.data_ptr(), cu.numel(), lo.data_ptr(), B, Sq, int(q_off), min(int(window_left), 1 << 30) if has_w else -1,
                                               _native.stream_ptr())
        _native.check(rc, "pt_row_lower_bounds")
        return lo
    key = (str(device), B, Sq, q_off, window_left if has_w else None)
    lo = _ROW_LO_CACHE.get(key) if cu_seqlens is None else None
    if lo is None:
        pos = torch.arange(Sq, device=device, dtype=torch.int64)
        lo = torch.zeros(Sq, device=device, dtype=torch.int64)
        if has_w:
            lo = torch.clamp(pos + q_off - int(window_left), min=0)
        if cu_seqlens is not None:
            cs = cu_seqlens.to(device=device, dtype=torch.int64)
            seg = torch.bucketize(pos, cs[1:], right=True).clamp_(max=cs.numel() - 2)
            lo = torch.maximum(lo, cs[seg])
        lo = lo.to(torch.int32).repeat(B).contiguous()
        if cu_seqlens is None:
            if len(_ROW_LO_CACHE) > 64:
                _ROW_LO_CACHE.clear()
            _ROW_LO_CACHE[key] = lo
    return lo


def _as_token_major(t: torch.Tensor) -> torch.Tensor:
    return t if _token_major(t) else t.contiguous()


def _aligned_gradient(do: torch.Tensor) -> torch.Tensor:
    """``do`` as the pass over its rows reads it, in 16-byte pieces. Unlike q, k and v it comes to no tensor map of the forward
    that would have refused a misaligned base or pitch, and ``contiguous()`` hands a contiguous piece of a larger gradient back
    as it is (one of a single row with whatever pitch it has)."""
    do = _as_token_major(do)
    return do if _token_major(do) else do.clone(memory_format=torch.contiguous_format)


def forward(q, k, v, scale: float, causal: bool, q_off: int, row_lo: Optional[torch.Tensor],
            sinks: Optional[torch.Tensor]) -> Tuple[torch.Tensor, torch.Tensor]:
    """Launch the forward kernel: returns ``out [B,Sq,Hq,Dv]`` bf16 and ``lse [B,Hq,Sq]`` fp32."""
    from .. import _native

    q, k, v = _as_token_major(q), _as_token_major(k), _as_token_major(v)
    B, Sq, Hq, D = q.shape
    Sk, Hkv, Dv = k.shape[1], k.shape[2], v.shape[-1]
    out = torch.empty((B, Sq, Hq, Dv), dtype=q.dtype, device=q.device)
    lse = torch.empty((B, Hq, Sq), dtype=torch.float32, device=q.device)
    sk = None if sinks is None else sinks.detach().float().contiguous()
    rc = _native.lib().pt_attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr(),
                                   _native.ptr(row_lo), _native.ptr(sk), B, Sq, Sk, Hq, Hkv, D, Dv, q.stride(1), k.stride(1),
                                   v.stride(1), out.stride(1), float(scale), int(bool(causal)), int(q_off),
                                   _native.stream_ptr())
    _native.check(rc, "pt_attn_fwd")
    return out, lse


def backward(do, q, k, v, out, lse, scale: float, causal: bool, q_off: int, row_lo: Optional[torch.Tensor]
             ) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor]:
    """Launch the backward kernels: returns ``dq, dk, dv`` (bf16) and ``delta [B,Hq,Sq]`` (fp32 row sums of dO*O,
    which the sink gradient needs)."""
    from .. import _native

    q, k, v, out, do = *(_as_token_major(t) for t in (q, k, v, out)), _aligned_gradient(do)
    lse = lse.contiguous()  # ring attention hands in halves of a longer sequence's statistics
    B, Sq, Hq, D = q.shape
    Sk, Hkv, Dv = k.shape[1], k.shape[2], v.shape[-1]
    # one zeroed buffer: the fp32 accumulators (dq over key tiles; dk / dv over the heads of a GQA group), then the row
    # statistics, padded by one tile because the kernel reads them in whole 128-row tiles
    nq, nk, ns = B * Sq * Hq * D, B * Sk * Hkv * D, B * Hq * Sq
    buf = torch.zeros(nq + 2 * nk + 2 * (ns + 128), dtype=torch.float32, device=q.device)
    delta, lse2 = buf[nq + 2 * nk:nq + 2 * nk + ns + 128], buf[nq + 2 * nk + ns + 128:]
    dq = torch.empty((B, Sq, Hq, D), dtype=q.dtype, device=q.device)
    dk = torch.empty((B, Sk, Hkv, D), dtype=k.dtype, device=q.device)
    dv = torch.empty((B, Sk, Hkv, Dv), dtype=v.dtype, device=q.device)
    rc = _native.lib().pt_attn_bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), do.data_ptr(), lse.data_ptr(),
                                   _native.ptr(row_lo), buf.data_ptr(), buf[nq:].data_ptr(), buf[nq + nk:].data_ptr(),
                                   dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), delta.data_ptr(), lse2.data_ptr(),
                                   B, Sq, Sk, Hq, Hkv, D, q.stride(1), k.stride(1), v.stride(1), out.stride(1), do.stride(1),
                                   float(scale), int(bool(causal)), int(q_off), _native.stream_ptr())
    _native.check(rc, "pt_attn_bwd")
    return dq, dk, dv, delta[:ns].view(B, Hq, Sq)


def backward_split(do, q, k, v, out, lse, scale: float, causal: bool, q_off: int, row_lo: Optional[torch.Tensor]
                   ) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor]:
    """:func:`backward` on the kernels that keep all 24 bits of P and dS (three bf16 terms each), for every head-dim pair
    of the forward kernel and any length. ``delta`` is a strided view."""
    from .. import _native

    q, k, v, out, do = *(_as_token_major(t) for t in (q, k, v, out)), _aligned_gradient(do)
    lse = lse.contiguous()
    B, Sq, Hq, D = q.shape
    Sk, Hkv, Dv = k.shape[1], k.shape[2], v.shape[-1]
    dev, Sp = q.device, (Sq + 3) // 4 * 4
    ns = B * Hq * Sp
    stats = torch.empty(2 * (ns + 128), dtype=torch.float32, device=dev)  # read in whole 64-row tiles: padded
    delta, lse2 = stats[:ns + 128], stats[ns + 128:]
    dq, dk, dv = (torch.empty(t.shape, dtype=t.dtype, device=dev) for t in (q, k, v))
    part = torch.empty(B * Sk * Hq * max(D, Dv), dtype=torch.float32, device=dev) if Hq != Hkv else None
    rc = _native.lib().pt_attn_bwd_split(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), do.data_ptr(), lse.data_ptr(),
                                         _native.ptr(row_lo), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), delta.data_ptr(),
                                         lse2.data_ptr(), _native.ptr(part), B, Sq, Sk, Hq, Hkv, D, Dv, q.stride(1), k.stride(1),
                                         v.stride(1), out.stride(1), do.stride(1), float(scale), int(bool(causal)), int(q_off),
                                         _native.stream_ptr())
    _native.check(rc, "pt_attn_bwd_split", launches=4 if part is None else 6)  # a group sum each for dK and dV
    return dq, dk, dv, delta[:ns].view(B, Hq, Sp)[..., :Sq]


def attention(q, k, v, causal, scale, window_left, sinks, cu_seqlens, return_lse=False, q_off: Optional[int] = None):
    """Attention of ``q [B,Sq,Hq,D]`` against ``k [B,Sk,Hkv,D]``, ``v [B,Sk,Hkv,Dv]`` on the own kernels (autograd-aware).
    ``q_off`` is the position of query 0 relative to key 0 (default ``Sk - Sq``: the last query sees the last key)."""
    B, Sq = q.shape[0], q.shape[1]
    Sk = k.shape[1]
    if q_off is None:
        q_off = Sk - Sq
    sc = float(scale) if scale is not None else q.shape[-1] ** -0.5
    row_lo = row_lower_bounds(B, Sq, q_off, window_left, cu_seqlens, q.device)
    from .. import _native

    reach = Sk if cu_seqlens is None else B * Sq // max(1, cu_seqlens.numel() - 1)  # about how many keys a query sees
    if window_left is not None and window_left >= 0:
        reach = min(reach, int(window_left) + 1)
    out, lse = _native.host().attention(q, k, v, sinks, row_lo, sc, bool(causal), int(q_off), min(int(reach), 2 ** 31 - 1))
    return (out, lse) if return_lse else out


def block_from_pointers(q: torch.Tensor, k_ptr: int, v_ptr: int, Sk: int, Hkv: int, scale: float
                        ) -> Tuple[torch.Tensor, torch.Tensor]:
    """Unmasked attention of ``q [1, Sq, Hq, D]`` against ``Sk`` keys/values stored token-major and contiguous
    (``[Sk, Hkv, D]`` bf16) at raw device addresses — which may lie in another GPU's published buffer: the kernel's
    TMA loads then fetch the block over NVLink tile by tile while it computes. Returns bf16 ``out`` and fp32 ``lse``."""
    from .. import _native

    q = _as_token_major(q)
    B, Sq, Hq, D = q.shape
    assert B == 1 and q.dtype == torch.bfloat16 and (D, D) in _DIMS
    out = torch.empty((1, Sq, Hq, D), dtype=q.dtype, device=q.device)
    lse = torch.empty((1, Hq, Sq), dtype=torch.float32, device=q.device)
    rc = _native.lib().pt_attn_fwd(q.data_ptr(), k_ptr, v_ptr, out.data_ptr(), lse.data_ptr(), None, None, 1, Sq, Sk, Hq, Hkv,
                                   D, D, q.stride(1), Hkv * D, Hkv * D, out.stride(1), float(scale), 0, 0,
                                   _native.stream_ptr())
    _native.check(rc, "pt_attn_fwd")
    return out, lse
