"""Token embedding lookup whose backward accumulates into the parameter's gradient buffer."""

from __future__ import annotations

import torch

from .. import _native
from .common import grad_buffer, sp, use_native
from .moe import gather_rows


class _EmbeddingFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, ids, weight):
        ctx.save_for_backward(ids)
        ctx.w_ref = weight
        flat = ids.reshape(-1)
        if weight.is_cuda and weight.dtype == torch.bfloat16 and weight.shape[1] % 8 == 0:
            out = gather_rows(weight.detach(), flat.int().contiguous())
        else:
            out = weight.detach()[flat]
        return out.view(*ids.shape, weight.shape[1])

    @staticmethod
    def backward(ctx, dy):
        (ids,) = ctx.saved_tensors
        w = ctx.w_ref
        g = grad_buffer(w)
        n, H = ids.numel(), dy.shape[-1]
        # fp32 gradients of bf16 rows; the additions into one row have no order, as those of index_add_
        if (use_native(dy) and dy.dtype == torch.bfloat16 and g.dtype == torch.float32 and g.device == dy.device == ids.device
                and ids.dtype == torch.int64 and H % 8 == 0 and g.is_contiguous() and g.data_ptr() % 16 == 0
                and not dy.requires_grad and not torch.are_deterministic_algorithms_enabled()):
            rows, flat = dy.reshape(n, H).contiguous(), ids.reshape(-1).contiguous()
            if rows.data_ptr() % 16 == 0:
                _native.check(_native.lib().pt_embedding_bwd(rows.data_ptr(), flat.data_ptr(), g.data_ptr(), n, H, g.shape[0], sp()), "pt_embedding_bwd")
                return None, None
        g.index_add_(0, ids.reshape(-1), dy.reshape(-1, dy.shape[-1]).to(g.dtype))
        return None, None


def embedding(ids: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    out = _EmbeddingFn.apply(ids, weight)
    return out


class Embedding(torch.nn.Embedding):
    def forward(self, ids: torch.Tensor) -> torch.Tensor:
        if torch.is_grad_enabled() and self.weight.requires_grad:
            # route through autograd with a dummy edge so backward() runs
            return _EmbeddingFn.apply(ids, self.weight)
        return _EmbeddingFn.apply(ids, self.weight)
