"""Router top-k with its softmax, forward and backward, in one kernel each.

* ``mode="softmax_topk"``: ``p = softmax(logits)`` in fp32, top-k of ``p``, optional renormalisation,
  times ``scale`` (Qwen3-MoE, DeepSeek-V2: pithtrain/models/qwen3_moe.py:81-89,
  pithtrain/models/deepseek_v2.py:149-164).
* ``mode="topk_softmax"``: top-k of the logits, softmax over the picked k (GPT-OSS:
  pithtrain/models/gpt_oss.py:176-182).

Returns ``(topk_weight[n,k] fp32, topk_idx[n,k] int32, probs[n,E] fp32 or None)``. ``probs`` is a
differentiable output so a load-balance loss can be built on it with ordinary autograd; its
gradient is folded into the same backward kernel.
"""

from __future__ import annotations

from typing import Optional, Tuple

import torch

from .. import _native
MODES = {"softmax_topk": 0, "topk_softmax": 1}


def router_topk_ref(logits, k, mode="softmax_topk", renorm=False, scale=1.0):
    lf = logits.float()
    if mode == "softmax_topk":
        p = lf.softmax(-1)
        w, idx = torch.topk(p, k, dim=-1)
        if renorm:
            w = w / w.sum(-1, keepdim=True)
        return w * scale, idx.int(), p
    v, idx = torch.topk(lf, k, dim=-1)
    return v.softmax(-1) * scale, idx.int(), None


def router_topk(logits: torch.Tensor, k: int, mode: str = "softmax_topk", renorm: bool = False,
                scale: float = 1.0) -> Tuple[torch.Tensor, torch.Tensor, Optional[torch.Tensor]]:
    n, E = logits.shape
    if logits.is_cuda and logits.dtype in (torch.float32, torch.bfloat16) and E <= 512 and k <= 16:
        m = MODES[mode]
        return _native.host().router(logits, None, k, m, renorm and m == 0, scale)
    return router_topk_ref(logits, k, mode, renorm, scale)


def _given_ref(logits, idx, renorm, scale):
    scores = logits.float().softmax(-1)
    w = scores.gather(-1, idx.long())
    if renorm:
        w = w / w.sum(-1, keepdim=True)
    return w * scale, idx.int(), scores


def router_replayed_ref(logits, k, replay, renorm=False, scale=1.0):
    return _given_ref(logits, replay(torch.topk(logits.float().softmax(-1), k, dim=-1).indices), renorm, scale)


def router_replayed(logits: torch.Tensor, k: int, replay, renorm: bool = False, scale: float = 1.0
                    ) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """:func:`router_topk` (``softmax_topk``) with the picks exchanged by ``replay(top-k indices) -> indices``: the weights are the
    softmax scores of the replayed experts. The indices are int64, or int32 for a ``replay`` with a true ``any_int``."""
    n, E = logits.shape
    if _native.on_current_device(logits) and logits.dtype in (torch.float32, torch.bfloat16) and E <= 512 and k <= 16 and n > 0:
        host = _native.host()
        picks = host.router_picks(logits, k)
        idx = replay(picks if getattr(replay, "any_int", False) else picks.long()).int().contiguous()
        if idx.device == logits.device and idx.dim() == 2 and idx.shape[0] == n and 0 < idx.shape[1] <= 16:
            w, idx, probs = host.router(logits, idx, k, 0, renorm, scale)
            return w, idx, probs
        return _given_ref(logits, idx, renorm, scale)
    return router_replayed_ref(logits, k, replay, renorm, scale)
