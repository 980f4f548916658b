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
