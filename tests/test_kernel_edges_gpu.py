"""Kernels at the sizes where they can go wrong: remainders, tile edges, the smallest and the largest of their range."""

import pytest
import torch

from pithtrain_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("G,ld,H", [(1, 8, 1), (3, 40, 33), (255, 256, 128), (257, 2048, 2048), (592, 100, 31)])
def test_colsum_accumulate(G, ld, H, dtype):
    torch.manual_seed(G)
    part = torch.randn(G, ld, device="cuda")
    dst = torch.randn(H, device="cuda").to(dtype)
    want = dst.double() + part[:, :H].double().sum(0)
    rc = _native.lib().pt_colsum_accumulate(part.data_ptr(), G, ld, H, dst.data_ptr(), int(dtype == torch.float32),
                                            _native.stream_ptr())
    _native.check(rc, "pt_colsum_accumulate")
    # fp32 sum of G terms of magnitude <= 5: |error| <= G * 5 * 2^-24 * (longest chain of additions, <= 16 + log2 G);
    # the bf16 result is rounded once more
    bound = G * 5 * 2.0 ** -24 * 24 + (want.abs() * 2.0 ** -8 if dtype == torch.bfloat16 else 0)
    assert ((dst.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("G,R,K", [(1, 8, 16), (2, 128, 128), (1, 130, 264), (3, 24, 136), (2, 272, 40), (1, 2880, 144)])
def test_quant_blocks_both_orientations(G, R, K):
    """Bytes and scales equal the plain tensor-op recipe, ragged edge tiles and unaligned pitches of W^T included."""
    from pithtrain_b200.ops.quant import quant_blocks, quant_blocks_ref

    torch.manual_seed(R)
    w = (torch.randn(G, R, K, device="cuda") * 0.02).bfloat16()
    q, s, qt, st = quant_blocks(w)
    q0, s0 = quant_blocks_ref(w)
    assert torch.equal(q.view(torch.uint8), q0.view(torch.uint8)) and torch.equal(s, s0)
    assert torch.equal(qt.view(torch.uint8), q0.transpose(1, 2).contiguous().view(torch.uint8))
    assert torch.equal(st, s0.transpose(1, 2).contiguous())
