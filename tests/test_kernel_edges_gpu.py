"""Kernels at the sizes where they can go wrong: remainders, tile edges, the smallest and the largest of their range."""

import pytest
import torch

from pithtrain_b200 import _native
from pithtrain_b200.ops import attention as A
from pithtrain_b200.ops import attention_native as N

pytestmark = pytest.mark.gpu


def _backward64(do, q, k, v, out, lse, scale, causal, q_off, row_lo):
    """The flash-attention backward formulas in 64 bits, from the same bf16 ``out`` and fp32 ``lse``."""
    B, Sq, Hq, D = q.shape
    Sk, Hkv = k.shape[1], k.shape[2]
    g = Hq // Hkv
    qf, dof = q.double().permute(0, 2, 1, 3), do.double().permute(0, 2, 1, 3)
    kf, vf = (t.double().permute(0, 2, 1, 3).repeat_interleave(g, dim=1) for t in (k, v))
    kp = torch.arange(Sk, device=q.device).view(1, 1, 1, Sk)
    qp = (torch.arange(Sq, device=q.device) + q_off).view(1, 1, Sq, 1)
    vis = torch.ones(1, 1, Sq, Sk, dtype=torch.bool, device=q.device)
    if causal:
        vis = vis & (kp <= qp)
    if row_lo is not None:
        vis = vis & (kp >= row_lo.view(B, 1, Sq, 1))
    safe = torch.where(torch.isinf(lse), torch.zeros_like(lse), lse).double()
    p = torch.exp(qf @ kf.mT * scale - safe[..., None]).masked_fill(~vis, 0.0)
    delta = (dof * out.double().permute(0, 2, 1, 3)).sum(-1)
    ds = p * (dof @ vf.mT - delta[..., None]) * scale
    dq = (ds @ kf).permute(0, 2, 1, 3)
    dk = (ds.mT @ qf).view(B, Hkv, g, Sk, D).sum(2).permute(0, 2, 1, 3)
    dv = (p.mT @ dof).view(B, Hkv, g, Sk, -1).sum(2).permute(0, 2, 1, 3)
    return dq, dk, dv, delta


# Rounding to bf16 is off by at most 2^-8 of a value (half a unit in the last of 8 bits); over many values the 2-norm of
# errors uniform over that half unit is at most 2^-8 / sqrt(3).
BF16_MAX, BF16_NORM = 2.0 ** -8, 2.0 ** -8 / 3 ** 0.5


def _rel(a, b):
    return float((a.double() - b).norm() / b.norm().clamp_min(1e-30))


@pytest.mark.parametrize("Dqk,Dv,Hq,Hkv", [(64, 64, 4, 2), (128, 128, 2, 2), (192, 128, 2, 2), (256, 256, 4, 1)])
@pytest.mark.parametrize("B,Sq,Sk,causal,window,docs", [
    (1, 1, 1, True, None, None), (2, 3, 3, True, None, None), (1, 63, 63, True, None, None), (2, 65, 65, True, None, None),
    (1, 127, 127, True, None, None), (2, 130, 130, True, None, None), (1, 257, 257, False, None, None),
    (1, 64, 320, True, None, None), (2, 96, 200, False, None, None), (1, 515, 515, True, 100, None),
    (1, 517, 517, True, None, [0, 1, 130, 131, 400, 517]), (1, 640, 640, True, 64, [0, 128, 129, 512, 640]),
    (2, 325, 325, True, 70, None), (3, 200, 200, True, None, [0, 1, 64, 130, 200]), (2, 66, 200, True, 40, None),
])
def test_attention_backward_split(Dqk, Dv, Hq, Hkv, B, Sq, Sk, causal, window, docs):
    """dq, dk, dv are the 64-bit gradients rounded to bf16: P and dS lose nothing on the way (rounding them too would show as
    3e-3)."""
    torch.manual_seed(Sq)
    q = torch.randn(B, Sq, Hq, Dqk, device="cuda").bfloat16()
    k, v = torch.randn(B, Sk, Hkv, Dqk, device="cuda").bfloat16(), torch.randn(B, Sk, Hkv, Dv, device="cuda").bfloat16()
    do = torch.randn(B, Sq, Hq, Dv, device="cuda").bfloat16()
    cu = None if docs is None else torch.tensor(docs, dtype=torch.int32, device="cuda")
    scale, q_off = Dqk ** -0.5, Sk - Sq
    row_lo = N.row_lower_bounds(B, Sq, q_off, window, cu, q.device)
    out, lse = N.forward(q, k, v, scale, causal, q_off, row_lo, None)
    got = N.backward_split(do, q, k, v, out, lse, scale, causal, q_off, row_lo)
    _native.check_status()
    want = _backward64(do, q, k, v, out, lse, scale, causal, q_off, row_lo)
    if Sq == 1 and Sk == 1:
        # one key: P = 1 and dS = dP - delta, which cancels up to the rounding of out (2^-8 of terms of size D^0.5 * 3)
        assert _rel(got[2], want[2]) < BF16_MAX
        assert (got[0].double() - want[0]).abs().max() < BF16_MAX * 3 * Dv ** 0.5 * scale * 4
        return
    for name, a, b in zip(("dq", "dk", "dv"), got, want):
        # fp32 accumulation and lse add less than 2^-12 to the rounding of the result
        assert _rel(a, b) < BF16_NORM + 2.0 ** -12, name
    assert _rel(got[3], want[3]) < 1e-5


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,S,Hq,Hkv,docs,window", [(1, 130, 148, 37, 1, None), (1, 130, 149, 149, 1, None), (5, 67, 64, 8, 1, None), (1, 130, 75, 25, 13, None),
                                                    (1, 259, 50, 10, 1, 40), (1, 3, 300, 60, 1, None), (2, 1025, 33, 11, 1, None), (2, 770, 43, 43, 1, None)])
def test_attention_backward_split_alone_and_paired(D, B, S, Hq, Hkv, docs, window):
    """On both sides of the lines between one CTA an SM and two (148 SMs: 148, 296, 592 CTAs), by the number of CTAs and of keys a query sees."""
    torch.manual_seed(S + Hq)
    q, k, v = (torch.randn(B, S, h, D, device="cuda").bfloat16().requires_grad_() for h in (Hq, Hkv, Hkv))
    cu = None if docs == 1 else torch.linspace(0, S, docs + 1).int().cuda()
    out, lse = N.attention(q, k, v, True, None, window, None, cu, return_lse=True)
    do = torch.randn_like(out)
    got = torch.autograd.grad(out, (q, k, v), do)
    row_lo = N.row_lower_bounds(B, S, 0, window, cu, q.device)
    with torch.no_grad():
        for a, b in zip(got, _backward64(do, q, k, v, out, lse, D ** -0.5, True, 0, row_lo)):
            assert _rel(a, b) <= BF16_NORM
    _native.check_status()


@pytest.mark.parametrize("Dqk,Dv,Hq,Hkv", [(64, 64, 2, 1), (128, 128, 2, 1), (192, 128, 1, 1), (256, 256, 1, 1)])
@pytest.mark.parametrize("Sq,docs", [(2113, 1), (2113, 40), (4201, 300), (2305, 2304)])
def test_attention_backward_split_finds_its_tiles(Dqk, Dv, Hq, Hkv, Sq, docs):
    """More than 32 tiles of 64 rows, so that the search for the last tile takes two rounds of probes; documents of one row
    upwards, many in one tile."""
    torch.manual_seed(docs)
    q, k = (torch.randn(1, Sq, h, Dqk, device="cuda").bfloat16() for h in (Hq, Hkv))
    v, do = torch.randn(1, Sq, Hkv, Dv, device="cuda").bfloat16(), torch.randn(1, Sq, Hq, Dv, device="cuda").bfloat16()
    cuts = sorted((torch.randperm(Sq - 1)[:docs - 1] + 1).tolist())
    cu = torch.tensor([0, *cuts, Sq], dtype=torch.int32, device="cuda")
    row_lo = N.row_lower_bounds(1, Sq, 0, None, cu, q.device)
    out, lse = N.forward(q, k, v, Dqk ** -0.5, True, 0, row_lo, None)
    got = N.backward_split(do, q, k, v, out, lse, Dqk ** -0.5, True, 0, row_lo)
    _native.check_status()
    want = _backward64(do, q, k, v, out, lse, Dqk ** -0.5, True, 0, row_lo)
    bound = BF16_NORM + 2.0 ** -12
    assert _rel(got[2], want[2]) < bound  # dv has no cancellation
    for a, b in zip(got[:2], want[:2]):
        # rows that see one key have dS = dP - delta = 0 up to the rounding of out, 2^-8 of terms of size 3 D^0.5
        slack = BF16_MAX * 3 * Dv ** 0.5 * Dqk ** -0.5 * 4 * (a.numel() * min(1.0, 2 * docs / Sq)) ** 0.5
        assert float((a.double() - b).norm()) < bound * float(b.norm()) + slack


@pytest.mark.parametrize("Dqk,Dv", [(64, 64), (128, 128), (192, 128), (256, 256)])
def test_attention_backward_split_holds_fp32_probabilities(Dqk, Dv):
    """The fp32 partials of dV for each query head, before anything is rounded to bf16. One tile of queries: 12 products of the
    tensor core into the accumulator, each cut off by at most 2^-24 of it, and an exponential good to 2^-22; P in two bf16 terms
    (2^-17) would show as 2e-6."""
    torch.manual_seed(Dqk)
    S, Hq, Hkv = 64, 4, 2
    q, k, v, do = (torch.randn(1, S, h, d, device="cuda").bfloat16() for h, d in ((Hq, Dqk), (Hkv, Dqk), (Hkv, Dv), (Hq, Dv)))
    scale = Dqk ** -0.5
    out, lse = N.forward(q, k, v, scale, True, 0, None, None)
    dq, dk, dv = (torch.empty_like(t) for t in (q, k, v))
    delta, lse2 = (torch.empty(Hq * S + 128, device="cuda") for _ in range(2))
    part = torch.empty(S * Hq * Dqk, device="cuda")  # holds dV's partials last
    rc = _native.lib().pt_attn_bwd_split(*(t.data_ptr() for t in (q, k, v, out, do, lse)), None,
                                         *(t.data_ptr() for t in (dq, dk, dv, delta, lse2, part)), 1, S, S, Hq, Hkv, Dqk, Dv,
                                         q.stride(1), k.stride(1), v.stride(1), out.stride(1), do.stride(1), scale, 1, 0, _native.stream_ptr())
    _native.check(rc, "pt_attn_bwd_split")
    _native.check_status()
    qd, dod, kd = (t.double().permute(0, 2, 1, 3) for t in (q, do, k.repeat_interleave(Hq // Hkv, 2)))
    p = torch.exp(qd @ kd.mT * scale - lse.double()[..., None]).tril()
    assert _rel(part[:S * Hq * Dv].view(1, S, Hq, Dv), (p.mT @ dod).permute(0, 2, 1, 3)) < 2.0 ** -20


def test_attention_backward_split_keeps_batch_entries_apart():
    """Rows past the end of a batch entry read as zero: an infinity in the next entry stays there."""
    q, k, v, do = (torch.randn(2, 70, 2, 256, device="cuda").bfloat16() for _ in range(4))
    for t in (q, k, v, do):
        t[1] = float("inf")
    out, lse = N.forward(q[:1], k[:1], v[:1], 0.0625, True, 0, None, None)
    out, lse = torch.cat([out, out]), torch.cat([lse, lse])
    got = N.backward_split(do, q, k, v, out, lse, 0.0625, True, 0, None)
    want = _backward64(do[:1], q[:1], k[:1], v[:1], out[:1], lse[:1], 0.0625, True, 0, None)
    for a, b in zip(got[:3], want):
        assert _rel(a[:1], b) < BF16_NORM + 2.0 ** -12


@pytest.mark.parametrize("S", [126, 1021])
def test_attention_with_odd_lengths_and_sinks(S):
    torch.manual_seed(S)
    q = torch.randn(1, S, 4, 128, device="cuda").bfloat16()
    k, v = (torch.randn(1, S, 2, 128, device="cuda").bfloat16() for _ in range(2))
    sinks, do = torch.randn(4, device="cuda").bfloat16(), torch.randn(1, S, 4, 128, device="cuda").bfloat16()

    def grads(fn):
        leaves = [t.detach().clone().requires_grad_() for t in (q, k, v, sinks)]
        return torch.autograd.grad(fn(*leaves), leaves, do)

    got = grads(lambda a, b, c, s: N.attention(a, b, c, True, None, 200, s, None))
    want = grads(lambda a, b, c, s: A.attention_ref(a, b, c, True, None, 200, s, None))
    _native.check_status()
    for a, b in zip(got, want):
        assert _rel(a, b.double()) < 1e-2  # the oracle differentiates an fp32 output, the kernels its bf16 rounding


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


def _delta_rule64(q, k, v, g, beta):
    """Token-by-token recurrence in 64 bits."""
    B, S, H, dk = q.shape
    state = torch.zeros(B, H, dk, v.shape[-1], dtype=torch.float64, device=q.device)
    outs = []
    for t in range(S):
        state = state * g[:, t].exp()[..., None, None]
        new = (v[:, t] - torch.einsum("bhkv,bhk->bhv", state, k[:, t])) * beta[:, t][..., None]
        state = state + k[:, t][..., None] * new[..., None, :]
        outs.append(torch.einsum("bhkv,bhk->bhv", state, q[:, t]) * dk ** -0.5)
    return torch.stack(outs, 1)


@pytest.mark.parametrize("B,S,H,strong", [(1, 1, 1, False), (2, 63, 2, False), (1, 64, 3, True), (1, 65, 2, False), (2, 130, 2, True),
                                          (1, 321, 4, False)])
def test_gated_delta_rule_fused(B, S, H, strong):
    """Outputs and all gradients of the fused kernels against the recurrence in 64 bits, q / k / v as slices of one projection;
    bf16 results carry one rounding, the fp32 gate gradients the error of fp32 sums."""
    from pithtrain_b200.ops.gated_delta_rule import gated_delta_rule

    torch.manual_seed(S)
    x = torch.randn(B, S, 3 * H * 128 + 8, device="cuda").bfloat16()
    q, k, v = (x[..., i * H * 128:(i + 1) * H * 128].view(B, S, H, 128) for i in range(3))
    q, k = (torch.nn.functional.normalize(t.float(), dim=-1).bfloat16() for t in (q, k))
    g = -torch.rand(B, S, H, device="cuda") * (6.0 if strong else 0.3)
    beta = torch.rand(B, S, H, device="cuda").bfloat16()
    do = torch.randn(B, S, H, 128, device="cuda").bfloat16()
    leaves = [t.detach().requires_grad_() for t in (q, k, v, g, beta)]
    assert S == 1 or leaves[2].stride(1) == x.stride(1)  # read in place
    o = gated_delta_rule(*leaves)
    got = torch.autograd.grad(o, leaves, do)
    wide = [t.detach().double().requires_grad_() for t in (q, k, v, g, beta)]
    ref = _delta_rule64(*wide)
    want = torch.autograd.grad(ref, wide, do.double())
    assert o.dtype == torch.bfloat16 and got[3].dtype == torch.float32 and got[4].dtype == torch.bfloat16
    assert _rel(o, ref.detach()) < BF16_NORM + 2.0 ** -12
    for name, a, b in zip(("dq", "dk", "dv", "dg", "dbeta"), got, want):
        if name == "dg":
            # a gate's gradient sums D^2 products that partly cancel: bounded against the size of its terms
            assert (a.double() - b).abs().max() < 1e-4 * b.abs().max().clamp_min(1.0), name
        else:
            assert _rel(a, b) < BF16_MAX, name


@pytest.mark.parametrize("bad", [float("nan"), float("-inf")])
@pytest.mark.parametrize("t", [0, 70, 199])
def test_gated_delta_rule_keeps_a_broken_gate_visible(t, bad):
    """A NaN or infinite log gate shows in every output that the tensor-op form (fp32 inputs) loses to it, in gradients of q, k,
    v, g and beta of that head, and nowhere in the other heads."""
    from pithtrain_b200.ops.gated_delta_rule import gated_delta_rule

    torch.manual_seed(t)
    S = 200
    q, k, v = (torch.nn.functional.normalize(torch.randn(1, S, 2, 128, device="cuda"), dim=-1).bfloat16() for _ in range(3))
    g, beta = -torch.rand(1, S, 2, device="cuda") * 0.3, torch.rand(1, S, 2, device="cuda")
    g[0, t, 1] = bad
    fine = {}
    for name, dtype in (("fused", torch.bfloat16), ("general", torch.float32)):
        leaves = [x.detach().to(dtype).requires_grad_() for x in (q, k, v)] + [x.clone().requires_grad_() for x in (g, beta)]
        o = gated_delta_rule(*leaves)
        grads = torch.autograd.grad(o, leaves, torch.ones_like(o))
        fine[name] = [torch.isfinite(x.detach()).view(S, 2, -1).all(-1) for x in (o, *grads)]
    assert torch.equal(fine["fused"][0], fine["general"][0])
    for got, want in zip(fine["fused"], fine["general"]):
        assert got[:, 0].all() and want[:, 0].all()
        assert not got[:, 1].all() and not want[:, 1].all()


def test_gated_delta_rule_with_gates_beyond_the_range_of_exp():
    """Gates that close a head entirely (e^-200 = 0) or grow its state (e^1 a step): as the tensor-op form."""
    from pithtrain_b200.ops.gated_delta_rule import gated_delta_rule

    torch.manual_seed(1)
    q, k, v = (torch.nn.functional.normalize(torch.randn(1, 130, 3, 128, device="cuda"), dim=-1).bfloat16() for _ in range(3))
    g = torch.tensor([-200.0, -0.1, 0.3], device="cuda").expand(1, 130, 3)
    beta = torch.rand(1, 130, 3, device="cuda")
    got, want = gated_delta_rule(q, k, v, g, beta), gated_delta_rule(q.float(), k.float(), v.float(), g, beta)
    for h in range(3):
        assert _rel(got[:, :, h], want[:, :, h].double()) < BF16_NORM + 2.0 ** -12, h


def _shifted(t, by=4):
    """The same values, contiguous, ``by`` elements into their storage."""
    return torch.cat([t.new_zeros(by), t.flatten()])[by:].view(t.shape)


def test_gated_delta_rule_on_misaligned_inputs():
    from pithtrain_b200.ops.gated_delta_rule import gated_delta_rule

    torch.manual_seed(2)
    ts = [torch.nn.functional.normalize(torch.randn(2, 67, 2, 128, device="cuda"), dim=-1).bfloat16() for _ in range(4)]
    g, beta = -torch.rand(2, 67, 2, device="cuda"), torch.rand(2, 67, 2, device="cuda").bfloat16()
    outs = []
    for move in (lambda t: t.clone(), _shifted):
        leaves = [move(t).requires_grad_() for t in (*ts[:3], g, beta)]
        o = gated_delta_rule(*leaves)
        outs.append([o, *torch.autograd.grad(o, leaves, move(ts[3]))])
    for a, b in zip(*outs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("elsewhere", [1, 2, 3, 4])
def test_gated_delta_rule_refuses_inputs_on_another_device(elsewhere):
    from pithtrain_b200.ops.gated_delta_rule import gated_delta_rule

    ts = [torch.rand(1, 9, 2, 128, device="cuda").bfloat16() for _ in range(3)] + [torch.rand(1, 9, 2, device="cuda") for _ in range(2)]
    ts[elsewhere] = ts[elsewhere].cpu()
    with pytest.raises(RuntimeError):
        gated_delta_rule(*ts)


@pytest.mark.parametrize("B,S,nk,nv", [(1, 1, 1, 1), (2, 3, 1, 2), (1, 31, 2, 2), (2, 33, 2, 4), (1, 97, 3, 9)])
def test_gdn_conv(B, S, nk, nv):
    """Convolution + SiLU + l2 norm + repetition and its gradients against tensor ops in 64 bits: one bf16 rounding each."""
    from pithtrain_b200.ops import gdn_mix

    F = torch.nn.functional
    torch.manual_seed(S)
    C = (2 * nk + nv) * 128
    x, w = torch.randn(B, S, C, device="cuda").bfloat16(), (torch.randn(C, 1, 4, device="cuda") * 0.4).bfloat16()
    go = [torch.randn(B, S, nv, 128, device="cuda").bfloat16() for _ in range(3)]
    xg, wp = x.clone().requires_grad_(), torch.nn.Parameter(w.clone())
    wp.main_grad = torch.zeros(w.shape, device="cuda")
    assert gdn_mix.conv_supported(xg, wp, nk, nv, 128, 128)
    got = gdn_mix.conv_qkv(xg, wp, nk, nv)
    torch.autograd.backward(got, go)
    xd, wd = x.double().requires_grad_(), w.double().requires_grad_()
    m = F.silu(F.conv1d(F.pad(xd.mT, (3, 0)), wd, groups=C)).mT
    q, k, v = m.split([nk * 128, nk * 128, nv * 128], -1)
    q, k = (F.normalize(t.reshape(B, S, nk, 128), dim=-1).repeat_interleave(nv // nk, 2) for t in (q, k))
    want = (q, k, v.reshape(B, S, nv, 128))
    torch.autograd.backward(want, [g.double() for g in go])
    for a, b in zip(got, want):
        assert _rel(a.detach(), b.detach()) < BF16_MAX
    assert _rel(xg.grad, xd.grad) < BF16_MAX
    assert _rel(wp.main_grad, wd.grad) < 1e-5


@pytest.mark.parametrize("rows", [1, 7, 8, 9, 20000])
def test_gdn_gated_norm(rows):
    from pithtrain_b200.ops import gdn_mix

    torch.manual_seed(rows)
    x, z, d = (torch.randn(rows, 128, device="cuda").bfloat16() for _ in range(3))
    w = (1 + 0.1 * torch.randn(128, device="cuda")).bfloat16()
    xg, zg, wp = x.clone().requires_grad_(), z.clone().requires_grad_(), torch.nn.Parameter(w.clone())
    wp.main_grad = torch.zeros(128, device="cuda")
    got = gdn_mix.gated_norm(xg, zg, wp, 1e-6)
    got.backward(d)
    xd, zd, wd = (t.double().requires_grad_() for t in (x, z, w))
    want = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * wd * torch.nn.functional.silu(zd)
    want.backward(d.double())
    for a, b in ((got.detach(), want.detach()), (xg.grad, xd.grad), (zg.grad, zd.grad)):
        assert _rel(a, b) < BF16_MAX
    assert _rel(wp.main_grad, wd.grad) < 1e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,E,k,renorm", [(1, 4, 1, True), (9, 16, 4, False), (257, 130, 6, True), (64, 512, 16, True)])
def test_router_replayed(n, E, k, renorm, dtype):
    """Weights, scores and logit gradients of replayed picks against the tensor-op form in 64 bits, repeated picks included."""
    from pithtrain_b200.ops.router import router_replayed

    torch.manual_seed(n)
    logits = (torch.randn(n, E, device="cuda") * 4).to(dtype)
    picks = torch.randint(0, E, (n, k), device="cuda")
    seen = []

    def replay(idx):
        seen.append(idx)
        return picks

    lg = logits.clone().requires_grad_()
    w, idx, probs = router_replayed(lg, k, replay, renorm, 2.5)
    dw, dp = torch.randn(n, k, device="cuda"), torch.randn(n, E, device="cuda")
    torch.autograd.backward((w, probs), (dw, dp))
    ld = logits.double().requires_grad_()
    p = ld.softmax(-1)
    want = p.gather(1, picks)
    want = (want / want.sum(-1, keepdim=True) if renorm else want) * 2.5
    torch.autograd.backward((want, p), (dw.double(), dp.double()))
    assert seen[0].dtype == torch.int64
    if dtype == torch.float32:
        assert torch.equal(seen[0], p.topk(k).indices)
    else:  # bf16 logits tie: other picks of the same scores, no pick twice
        assert torch.equal(ld.detach().gather(1, seen[0]), ld.detach().topk(k).values)
        assert all(r.unique().numel() == k for r in seen[0])
    assert torch.equal(idx.long(), picks)
    assert _rel(w.detach(), want.detach()) < 1e-6 and _rel(probs.detach(), p.detach()) < 1e-6
    # a logit's gradient is p times a difference that may cancel: fp32 error of its terms, then the rounding of the result
    size = 2.5 * float(dw.abs().max()) * k + float(dp.abs().max())
    assert ((lg.grad.double() - ld.grad).abs() <= 1e-6 * size + (BF16_MAX * ld.grad.abs() if dtype == torch.bfloat16 else 0)).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_router_replayed_keeps_nan(dtype):
    """A NaN or +inf logit, or a row of -inf, spoils its own row as the library softmax has it, and no other; forward and backward."""
    from pithtrain_b200.ops.router import router_replayed

    torch.manual_seed(3)
    logits = torch.randn(6, 40, device="cuda").to(dtype)
    logits[1, 35], logits[2], logits[3, 0], logits[4, 7] = float("nan"), float("-inf"), float("inf"), float("-inf")
    picks = torch.tensor([[0, 7, 35]], device="cuda").repeat(6, 1)
    lg = logits.clone().requires_grad_()
    w, _, probs = router_replayed(lg, 3, lambda idx: picks, True)
    w.sum().backward()
    ld = logits.double().requires_grad_()
    want = ld.softmax(-1)
    wd = want.gather(1, picks) / want.gather(1, picks).sum(-1, keepdim=True)
    wd.sum().backward()
    assert torch.equal(probs.isnan(), want.isnan()) and torch.equal(w.isnan(), wd.isnan()) and torch.equal(lg.grad.isnan(), ld.grad.isnan())
    ok = [0, 4, 5]
    assert _rel(probs[ok].detach(), want[ok].detach()) < 1e-6 and float(probs[4, 7]) == 0.0


@pytest.mark.parametrize("E,k", [(4, 4), (40, 3), (512, 16)])
def test_router_picks_of_a_nan_row_are_experts(E, k):
    """The replay, and the natural router's callers, get k different experts of weight NaN for a row without an order."""
    from pithtrain_b200.ops.router import router_replayed, router_topk

    logits = torch.randn(5, E, device="cuda")
    logits[1, E - 1], logits[3] = float("nan"), float("-inf")
    w, idx, _ = router_replayed(logits, k, lambda i: i, True)
    w0, idx0, _ = router_topk(logits, k, "softmax_topk", True)
    assert torch.equal(idx, idx0) and torch.equal(w.isnan(), w0.isnan())
    assert ((idx >= 0) & (idx < E)).all() and all(r.unique().numel() == k for r in idx)
    assert torch.equal(w.isnan().all(-1), torch.tensor([False, True, False, True, False], device="cuda"))


@pytest.mark.parametrize("renorm", [False, True])
@pytest.mark.parametrize("E", [16, 40, 512])
def test_router_replayed_picks_out_of_range(E, renorm):
    """A pick outside [0, E) has the weight NaN (renormalised, so has its row) and is read nowhere; other rows are untouched."""
    from pithtrain_b200.ops.router import router_replayed

    torch.manual_seed(E)
    logits = torch.randn(4, E, device="cuda")
    picks = torch.tensor([[0, 1, 2], [3, -1, 4], [E, 5, 6], [7, 8, E - 1]], device="cuda")
    lg, ld = logits.clone().requires_grad_(), logits.double().requires_grad_()
    w, idx, probs = router_replayed(lg, 3, lambda i: picks, renorm)
    out = torch.zeros_like(w, dtype=torch.bool)
    out[1, 1] = out[2, 0] = True
    assert torch.equal(idx.long(), picks) and torch.equal(w.isnan(), out.any(-1, keepdim=True).expand_as(out) if renorm else out)
    w[[0, 3]].sum(1).dot(torch.tensor([1.0, 2.0], device="cuda")).backward()
    p = ld.softmax(-1)
    wd = p.gather(1, picks.clamp(0, E - 1))
    wd = wd / wd.sum(-1, keepdim=True) if renorm else wd
    wd[[0, 3]].sum(1).dot(torch.tensor([1.0, 2.0], dtype=torch.float64, device="cuda")).backward()
    assert _rel(probs.detach(), p.detach()) < 1e-6 and _rel(w[[0, 3]].detach(), wd[[0, 3]].detach()) < 1e-6
    assert (lg.grad.double() - ld.grad)[[0, 3]].abs().max() <= 1e-6 * 2 * 3
    if not renorm:  # the weights that were not used carry no gradient
        assert not lg.grad[[1, 2]].any()


def test_router_replayed_refuses_picks_on_another_device():
    from pithtrain_b200.ops.router import router_replayed

    with pytest.raises(RuntimeError):
        router_replayed(torch.randn(3, 8, device="cuda"), 2, lambda idx: idx.cpu())


@pytest.mark.parametrize("k", [1, 3, 4, 6, 8])
@pytest.mark.parametrize("n,H", [(1, 8), (3, 264), (64, 2048), (3072, 264), (3073, 264), (5000, 512)])
def test_combine_rows(n, H, k):
    from pithtrain_b200.ops.moe import combine_rows

    torch.manual_seed(n)
    y = torch.randn(2 * n + 1, H, device="cuda").bfloat16()
    rows = torch.randint(-1, 2 * n + 1, (n * k,), device="cuda", dtype=torch.int32)  # -1: a slot whose expert is elsewhere
    w, res = torch.rand(n, k, device="cuda"), torch.randn(n, H, device="cuda").bfloat16()
    r = rows.view(n, k).long()
    picked = y.double()[r.clamp(min=0)] * (r >= 0)[..., None]
    for got, want in ((combine_rows(y, rows, k), picked.sum(1)), (combine_rows(y, rows, k, w, res), (picked * w.double()[..., None]).sum(1) + res.double())):
        # fp32 sums of k + 1 terms, one bf16 rounding
        assert ((got.double() - want).abs() <= BF16_MAX * want.abs() + 2.0 ** -20 * (k + 1) * 5).all()


@pytest.mark.parametrize("n,H,k", [(37, 2056, 5), (300, 2880, 4), (40, 4104, 8), (3, 12296, 2), (700, 64, 40), (2500, 256, 33), (65, 72, 16)])
def test_combine_rows_runs_and_slices(n, H, k):
    """Rows wider than one block's columns, runs of tokens past several loads of 32 indices, tokens of more slots than one load, and
    tokens without a row; an absent row is skipped, not multiplied: infinities next to it stay out."""
    from pithtrain_b200.ops.moe import combine_rows

    torch.manual_seed(n)
    y = torch.randn(2 * n, H, device="cuda").bfloat16()
    y[0] = float("inf")
    rows = torch.randint(1, 2 * n, (n, k), device="cuda", dtype=torch.int32)
    rows[torch.rand(n, k, device="cuda") < 0.3] = -1
    rows[:: 5] = -1
    w = torch.rand(n, k, device="cuda")
    w[rows < 0] = float("nan")
    got = combine_rows(y, rows.reshape(-1), k, w).double()
    want = torch.zeros(n, H, device="cuda", dtype=torch.double)
    for j in range(k):
        want += torch.where(rows[:, j : j + 1] >= 0, y[rows[:, j].long().clamp(min=0)].double() * w[:, j : j + 1].double(), 0.0)
    # fp32 sums of k terms below 5, one bf16 rounding
    assert ((got - want).abs() <= BF16_MAX * want.abs() + 2.0 ** -24 * k * k * 5).all()
    assert (got[::5] == 0).all()


@pytest.mark.parametrize("n,H,k", [(1535, 8, 3), (1536, 8, 3), (1536, 344, 3), (2559, 2056, 1), (2560, 2056, 1), (3072, 2304, 2), (3073, 2304, 2), (3073, 2312, 2),
                                   (3073, 4104, 2), (4096, 768, 4), (4097, 768, 4), (4097, 1536, 3), (4097, 72, 40), (4097, 264, 12), (20001, 264, 1)])
def test_combine_rows_of_either_kernel(n, H, k):
    """On both sides of the lines between the ring and a warp a token."""
    test_combine_rows_runs_and_slices(n, H, k)


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("sizes,N,K", [([16], 8, 8), ([0, 16, 80], 136, 40), ([48, 0, 0, 64], 264, 296), ([32] * 40, 392, 776)])
def test_grouped_weight_gradient_into_fp32(sizes, N, K, pair):
    """The prefetched read-modify-write epilogue: ragged tiles, empty groups (left alone), more tiles than CTAs, reproducible."""
    from pithtrain_b200.ops import gemm as G

    torch.manual_seed(N)
    o = [0]
    for s in sizes:
        o.append(o[-1] + s)
    offs = torch.tensor(o, dtype=torch.int32, device="cuda")
    mk = lambda c: torch.randn(o[-1] + 16, c, device="cuda").bfloat16()  # noqa: E731
    ops = [(mk(N), mk(K)) for _ in range(1 + pair)]
    start = torch.randn(len(sizes), N, K, device="cuda")
    want = start.double()
    for dy, x in ops:
        for g in range(len(sizes)):
            want[g] += dy[o[g]:o[g + 1]].double().T @ x[o[g]:o[g + 1]].double()
    outs = []
    for _ in range(2):
        out = start.clone()
        if pair:
            G.grouped_gemm_tn_pair(*ops[0], offs, *ops[1], offs, out)
        else:
            G.grouped_gemm_tn(*ops[0], offs, out, accumulate=True)
        _native.check_status()
        outs.append(out)
    # fp32 accumulation of at most 2 x 80 products of size < 25
    assert (outs[0].double() - want).abs().max() < 2.0 ** -24 * 160 * 25 * 2
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("positions", [False, True])
@pytest.mark.parametrize("n,S,H,dn,dr,dv", [(1, 1, 1, 8, 16, 8), (6, 3, 2, 128, 64, 128), (67, 67, 16, 128, 64, 128), (10, 5, 3, 24, 32, 40)])
def test_mla_assembly(n, S, H, dn, dr, dv, positions):
    from pithtrain_b200.ops import mla

    torch.manual_seed(n)
    wide = torch.randn(n, H * (dn + dr) + 40 + dr, device="cuda").bfloat16()  # q | latent | k_pe, as the fused projection writes them
    kv = torch.randn(n, H * (dn + dv), device="cuda").bfloat16()
    ang = torch.rand(S + 3, dr // 2, device="cuda") * 6
    cos, sin = (torch.cat([f(ang)] * 2, -1).bfloat16() for f in (torch.cos, torch.sin))
    pos = torch.randint(0, S + 3, (n,), device="cuda") if positions else None
    go = [torch.randn(n, H, d, device="cuda").bfloat16() for d in (dn + dr, dn + dr, dv)]
    assert mla.supported(wide, cos, H, dn, dr, dv)

    def leaves(dtype):
        return [t.to(dtype).requires_grad_() for t in (wide.clone(), kv.clone())]

    wl, kl = leaves(torch.bfloat16)
    q, lat, kp = mla.split_columns(wl, (H * (dn + dr), 40, dr))
    got = mla.mla_assemble(q, kp, kl, cos, sin, pos, S, H, dn, dr, dv)
    torch.autograd.backward((*got, lat), (*go, torch.ones_like(lat)))
    wd, kd = leaves(torch.float64)
    p = pos if positions else torch.arange(n, device="cuda") % S
    c, s = cos[p].double()[:, None], sin[p].double()[:, None]

    def rope(t):
        t = t.unflatten(-1, (dr // 2, 2)).transpose(-1, -2).flatten(-2)
        return t * c + torch.cat([-t[..., dr // 2:], t[..., : dr // 2]], -1) * s

    qd, ld, pd = wd.split((H * (dn + dr), 40, dr), -1)
    qd, kvd = qd.view(n, H, -1), kd.view(n, H, -1)
    want = (torch.cat([qd[..., :dn], rope(qd[..., dn:])], -1), torch.cat([kvd[..., :dn], rope(pd[:, None]).expand(-1, H, -1)], -1), kvd[..., dn:])
    torch.autograd.backward((*want, ld), (*(g.double() for g in go), torch.ones_like(ld)))
    for a, b in ((*zip(got, want), (wl.grad, wd.grad), (kl.grad, kd.grad))):
        # a rotation of two terms in fp32 (a sum of H of them for the shared key), rounded once
        a, b = a.detach().double(), b.detach()
        assert ((a - b).abs() <= BF16_MAX * b.abs() + 1e-6 * H * 5).all()


def test_mla_assembly_on_misaligned_inputs():
    from pithtrain_b200.ops import mla

    torch.manual_seed(6)
    q, kp, kv = (torch.randn(3, c, device="cuda").bfloat16() for c in (2 * 192, 64, 2 * 256))
    cos, sin = (torch.rand(3, 64, device="cuda").bfloat16() for _ in range(2))
    got = mla.mla_assemble(*(_shifted(t) for t in (q, kp, kv)), cos, sin, None, 3, 2, 128, 64, 128)
    for a, b in zip(got, mla.mla_assemble(q, kp, kv, cos, sin, None, 3, 2, 128, 64, 128)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("S,Dqk,Dv", [(67, 128, 128), (128, 192, 128), (64, 256, 256), (68, 64, 64)])
def test_attention_backward_of_a_misaligned_gradient(S, Dqk, Dv):
    """A contiguous piece of a larger gradient that starts 8 bytes into it."""
    torch.manual_seed(7)
    q, k, v, do = (torch.randn(1, S, 2, d, device="cuda").bfloat16() for d in (Dqk, Dqk, Dv, Dv))
    leaves = [t.requires_grad_() for t in (q, k, v)]
    out = N.attention(*leaves, True, None, None, None, None)
    for a, b in zip(torch.autograd.grad(out, leaves, _shifted(do), retain_graph=True), torch.autograd.grad(out, leaves, do)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("sizes", [[16], [0, 48, 16], [272, 0, 16, 528]])
@pytest.mark.parametrize("H", [8, 264, 2880])
def test_segment_sum_and_row_bias_dot(sizes, H):
    from pithtrain_b200.ops.moe import row_bias_dot, segment_sum

    torch.manual_seed(H)
    o = [0]
    for s in sizes:
        o.append(o[-1] + s)
    R, E = o[-1] + 32, len(sizes)
    offs = torch.tensor(o, dtype=torch.int32, device="cuda")
    x, bias, w = torch.randn(R, H, device="cuda").bfloat16(), torch.randn(E, H, device="cuda").bfloat16(), torch.rand(R, device="cuda")
    slots = torch.full((R,), -1, dtype=torch.int32, device="cuda")
    slots[: o[-1]] = torch.randperm(o[-1], device="cuda").int()
    slots[: o[-1] : 7] = -1
    group = torch.cat([torch.full((s,), g, device="cuda") for g, s in enumerate(sizes)])
    for t in (x, x.float()):
        for rw in (None, w):
            want = torch.zeros(E, H, dtype=torch.float64, device="cuda")
            want.index_add_(0, group, t[: o[-1]].double() * (1.0 if rw is None else rw[: o[-1], None].double()))
            got = segment_sum(t, offs, E, rw)
            assert (got.double() - want).abs().max() < 2.0 ** -24 * max(sizes) * 5 * 24
    dw = torch.randn(o[-1], device="cuda")
    want = dw.double()
    live = slots[: o[-1]] >= 0
    want[slots[: o[-1]][live].long()] += (x[: o[-1]][live].double() * bias[group[live]].double()).sum(-1)
    row_bias_dot(x, bias, offs, slots, dw, offs[E:E + 1])
    assert (dw.double() - want).abs().max() < 2.0 ** -24 * H * 25 * 16


@pytest.mark.parametrize("biased", [False, True])
def test_experts_without_tokens(biased):
    """A rank of an expert-parallel group that receives nothing: only pad rows, and no slot that they could take a weight from."""
    from pithtrain_b200.ops import moe as M

    k, E, H, I = 2, 4, 128, 64
    mk = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    x, w = mk(0, H).requires_grad_(), torch.rand(0, k, device="cuda").requires_grad_()
    g1, g2 = torch.zeros(E, 2 * I, H, device="cuda"), torch.zeros(E, H, I, device="cuda")
    b1, b2 = (torch.nn.Parameter(mk(E, c)) for c in (2 * I, H)) if biased else (None, None)
    ew = M.ExpertWeights(mk(E, 2 * I, H), mk(E, H, I), lambda: g1, lambda: g2, b1=b1, b2=b2)
    out = M.moe_experts(x, w, torch.zeros(0, k, dtype=torch.int32, device="cuda"), ew)
    out.backward(torch.ones_like(out))
    _native.check_status()
    assert out.shape == x.grad.shape == (0, H) and w.grad.shape == (0, k)
    assert all(not t.any() for t in (g1, g2, *((b1.grad, b2.grad) if biased else ())))


@pytest.mark.parametrize("window", [None, 0, 5, 300])
@pytest.mark.parametrize("docs", [[0, 1], [0, 7, 7, 8, 300], [0, 128, 256, 300], [0, 100, 200]])
def test_row_lower_bounds(docs, window):
    """Against the tensor-op form on the CPU: empty documents, rows past the last boundary, int64 boundaries."""
    for dtype in (torch.int32, torch.int64):
        cu = torch.tensor(docs, dtype=dtype)
        for Sq in (docs[-1], 300):
            got = N.row_lower_bounds(1, Sq, 0, window, cu.cuda(), torch.device("cuda", 0))
            assert torch.equal(got.cpu(), N.row_lower_bounds(1, Sq, 0, window, cu, torch.device("cpu")))


@pytest.mark.parametrize("shape", [(8, 8), (3, 8, 40), (5, 72, 24), (2, 264, 136), (1, 1024, 2048), (2, 12, 20), (4, 2, 4)])
@pytest.mark.parametrize("gdt,bdt", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32), (torch.float32, torch.bfloat16)])
def test_muon_update_with_fused_norm(shape, gdt, bdt):
    """The optimizer's step against the same step on tensor operations. The momentum is the same arithmetic in fp32; the
    scales differ from a separate norm's by its summation order, which moves a bf16 scale by one step at most: 2^-8 of the
    Gram matrix and of the first factor, and the iteration (derivative of its quintic at most a = 3.4445 a step, near 1 once
    converged) keeps that within 2^-8 * 3 of the update's size, added to the bf16 rounding of the weights."""
    from pithtrain_b200.modules.optimizer import Muon, muon_scale_factor, zeropower_via_newtonschulz5

    torch.manual_seed(5)
    w0 = torch.randn(shape, device="cuda").bfloat16()
    g, buf = torch.randn(shape, device="cuda").to(gdt), torch.randn(shape, device="cuda").to(bdt)
    if len(shape) == 3 and shape[0] > 2:
        g[1], buf[1] = 0, 0  # an expert without tokens: norm 0
    w, b1 = w0.clone(), buf.clone()
    opt = Muon([torch.nn.Parameter(w)], lr=0.1, momentum_dtype=bdt)
    opt._update_chunk(w.view(-1, *shape[-2:]), g.view(-1, *shape[-2:]), b1.view(-1, *shape[-2:]), 0.95, 0.1, 0.0)
    b32 = buf.float() * 0.95 + 0.05 * g.float()
    torch.testing.assert_close(b1.float(), b32.to(bdt).float(), rtol=2 ** -7 if bdt == torch.bfloat16 else 1e-6, atol=1e-6)  # one step of the type
    upd = (0.05 * g.float() + 0.95 * b32).bfloat16()
    step = 0.1 * muon_scale_factor(*shape[-2:]) * zeropower_via_newtonschulz5(upd).float()
    want, got = w0.float() - step, w.float()
    assert torch.isfinite(got).all()
    bound = 3 * BF16_MAX * float(step.norm()) + BF16_NORM * float(want.norm()) * 2
    assert float((got - want).norm()) <= bound


@pytest.mark.parametrize("M,N,K", [(1, 512, 8), (255, 776, 264), (257, 1032, 520), (1024, 520, 256), (1032, 8, 1032), (1999, 520, 264), (2056, 264, 776)])
def test_dense_products_on_cta_pairs(M, N, K):
    """Input and weight gradients at the edges of the 256-wide tiles and of the 64-long reduction blocks, against 64 bits: one
    rounding of the result on top of fp32 sums. The tensor core cuts each of its additions off (about n / 64 of 2^-24 a sum of n
    terms, measured 1e-9 n); ``fp32_sums`` has to stay within what the library's fp32 product shows."""
    from pithtrain_b200.ops import gemm as G
    from pithtrain_b200.ops.linear import _wgrad_into

    torch.manual_seed(M)
    dy, x, w = (torch.randn(s, device="cuda").bfloat16() for s in ((M, N), (M, K), (N, K)))
    rel = lambda a, b: float((a.double() - b).norm() / b.norm())  # noqa: E731
    # a rounding is at most 2^-8 of its value; the 2-norm's bound needs values enough to average over
    assert rel(G.gemm_nn(dy, w), dy.double() @ w.double()) <= (BF16_NORM if M * K > 64 else BF16_MAX)
    want = dy.double().t() @ x.double()
    assert rel(G.gemm_tn(dy, x, out=torch.zeros(N, K, device="cuda"), accumulate=True), want) <= 6e-8 + 2e-9 * M
    simt = rel(dy.float().t() @ x.float(), want)
    got = G.gemm_tn(dy, x, out=torch.zeros(N, K, device="cuda"), accumulate=True, fp32_sums=True)
    assert rel(got, want) <= max(simt, 1.5e-7)  # 128 rows a sum of the tensor core
    start = torch.randn(N, K, device="cuda")
    for target in (start.clone(), start.bfloat16()):
        before = target.double()
        _wgrad_into(dy, x, target)
        sum_ = before + want
        bound = 2e-7 + 2e-9 * M if target.dtype == torch.float32 else 2 * BF16_NORM  # the product and the sum are rounded
        assert rel(target, sum_) <= bound
    _native.check_status()


@pytest.mark.parametrize("shape", [(8, 8), (3, 8, 520), (2, 520, 8), (2, 248, 264), (1, 264, 248), (3, 256, 256), (2, 512, 776), (1, 1032, 520)])
def test_newton_schulz_products(shape):
    """Against the iteration in 64 bits, at the edges of the 256-wide tiles and of their mirrored halves. The kernels round the
    Gram matrices, the polynomial and the factors to bf16 once each, the tensor operations up to three times, so they may not be
    further off than those; 5 % for chance, since both errors are sums over random roundings."""
    from pithtrain_b200.modules.optimizer import _newton_schulz, zeropower_via_newtonschulz5

    torch.manual_seed(11)
    G = torch.randn(shape, device="cuda").bfloat16()
    before = G.clone()
    got, ops = zeropower_via_newtonschulz5(G), _newton_schulz(G, 5)
    _native.check_status()
    assert torch.equal(G, before) and got.shape == G.shape and got.dtype == torch.bfloat16
    X = G.double() / (torch.linalg.vector_norm(G.double(), dim=(-2, -1), keepdim=True) + 1e-7)
    for _ in range(5):
        A = X @ X.mT if shape[-2] <= shape[-1] else X.mT @ X
        B = -4.7750 * A + 2.0315 * A @ A
        X = 3.4445 * X + (B @ X if shape[-2] <= shape[-1] else X @ B)
    assert float((got.double() - X).norm()) <= 1.05 * float((ops.double() - X).norm())


def test_newton_schulz_under_transforms():
    """Autograd, forward mode and vmap see the tensor operations."""
    from pithtrain_b200.modules.optimizer import _newton_schulz, zeropower_via_newtonschulz5

    torch.manual_seed(13)
    G = torch.randn(2, 16, 24, device="cuda").bfloat16()
    leaf = G.clone().requires_grad_()
    assert torch.equal(torch.autograd.grad(zeropower_via_newtonschulz5(leaf).sum(), leaf)[0],
                       torch.autograd.grad(_newton_schulz(leaf, 5).sum(), leaf)[0])
    assert torch.equal(torch.func.vmap(zeropower_via_newtonschulz5)(G), torch.func.vmap(lambda g: _newton_schulz(g, 5))(G))
    one = torch.ones_like(G)
    assert torch.equal(torch.func.jvp(zeropower_via_newtonschulz5, (G,), (one,))[1],
                       torch.func.jvp(lambda g: _newton_schulz(g, 5), (G,), (one,))[1])


def test_muon_stacks_matrices_of_one_shape():
    """Parameters of one shape are orthogonalised together, others by themselves; both as one at a time."""
    from pithtrain_b200.modules.optimizer import Muon

    torch.manual_seed(12)
    shapes = [(64, 136), (64, 136), (3, 64, 136), (136, 64), (20, 12), (64, 136)]
    weights = [torch.randn(s, device="cuda").bfloat16() for s in shapes]
    grads = [torch.randn(s, device="cuda") for s in shapes]

    def run(groups, **kw):
        params = [torch.nn.Parameter(w.clone()) for w in weights]
        for p, g in zip(params, grads):
            p.main_grad = g
        for idx in groups:
            Muon([params[i] for i in idx], lr=0.1, **kw).step()
        _native.check_status()
        return params

    together = run([range(6)])
    for other in (run([[i] for i in range(6)]), run([range(6)], max_chunk_elems=2 * 64 * 136)):
        assert all(torch.equal(a, b) for a, b in zip(together, other))


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("n,E,k", [(1, 1, 1), (3, 4, 8), (257, 130, 6), (5000, 512, 16)])
def test_balanced_replay(n, E, k, dtype):
    from pithtrain_b200.modules.load_balance import force_balance

    picks = torch.zeros(n, k, dtype=dtype)
    got = force_balance(E)(picks.cuda())
    assert got.dtype == dtype and torch.equal(got.cpu(), force_balance(E)(picks))


@pytest.mark.parametrize("Hq,Hkv,D,R", [(1, 1, 64, 16), (3, 1, 64, 64), (4, 2, 128, 32), (2, 1, 256, 64), (5, 2, 256, 256)])
@pytest.mark.parametrize("n,view", [(1, False), (37, False), (515, True)])
def test_gated_attention_passes(n, view, Hq, Hkv, D, R):
    """Values and gradients against 64 bits: one bf16 rounding on each value; the weight sums are fp32."""
    from pithtrain_b200.ops import gated_attn as GA

    torch.manual_seed(n + D)
    C = 2 * (Hq + Hkv) * D
    lo = 8 if view else 0
    a = torch.randn(n, C + lo, device="cuda").bfloat16().requires_grad_()
    qw, kw = (torch.nn.Parameter((torch.randn(D, device="cuda") * 0.2).bfloat16()) for _ in range(2))
    for w in (qw, kw):
        w.main_grad = torch.ones(D, device="cuda")
    ang = torch.rand(n, R, device="cuda") * 6
    cos, sin = ang.cos().bfloat16(), ang.sin().bfloat16()
    assert GA.gated_attn_supported(a[:, lo:], qw, kw, R, Hq, Hkv, D)
    q, k, v, gate = GA.gated_attn_pre(a[:, lo:], qw, kw, cos, sin, Hq, Hkv, D, 1e-6)
    o = torch.randn(n, Hq, D, device="cuda").bfloat16().requires_grad_()
    y = GA.gated_attn_post(o, gate)

    a64, o64 = a.detach().double().requires_grad_(), o.detach().double().requires_grad_()
    w64 = [w.detach().double().requires_grad_() for w in (qw, kw)]
    x = a64[:, lo:]
    qg = x[:, :2 * Hq * D].view(n, Hq, 2, D)

    def normed(t, w):
        t = t * (t.pow(2).mean(-1, keepdim=True) + 1e-6).rsqrt() * (1 + w)
        r, c, s = t[..., :R], cos.double()[:, None], sin.double()[:, None]
        return torch.cat([r * c + torch.cat([-r[..., R // 2:], r[..., :R // 2]], -1) * s, t[..., R:]], -1)

    wants = (normed(qg[:, :, 0], w64[0]), normed(x[:, 2 * Hq * D:(2 * Hq + Hkv) * D].view(n, Hkv, D), w64[1]),
             x[:, (2 * Hq + Hkv) * D:].view(n, Hkv, D), o64 * qg[:, :, 1].sigmoid())
    ds = [torch.randn_like(t) for t in (q, k, v, y)]
    torch.autograd.backward((q, k, v, y), ds)
    torch.autograd.backward(wants, [d.double() for d in ds])
    # every result is rounded to bf16 once (the gate's gradient by its kernel, then copied)
    for got, want in list(zip((q, k, v, y), wants)) + [(o.grad, o64.grad), (a.grad, a64.grad)]:
        assert ((got.detach().double() - want.detach()).abs() <= BF16_MAX * want.detach().abs() + 1e-5 * want.detach().abs().max()).all()
    for w, d in zip((qw, kw), w64):
        assert _rel(w.main_grad - 1, d.grad) < 1e-5


@pytest.mark.parametrize("Hq,Hkv,D", [(1, 1, 64), (5, 1, 64), (4, 2, 128), (7, 7, 128)])
@pytest.mark.parametrize("n,pad,norm,with_dv", [(1, 0, True, True), (33, 8, True, True), (1030, 0, False, True), (600, 0, True, False)])
def test_qk_norm_rope_backward(n, pad, norm, with_dv, Hq, Hkv, D):
    """Gradients of the packed projection against 64 bits, rounded once; v's gradient is a copy, or zero if none reached it. The
    rotated and normalised value is rounded once more inside (before the rotation), which the gradient does not see."""
    from pithtrain_b200.ops.rope import qk_norm_rope

    torch.manual_seed(n)
    C = (Hq + 2 * Hkv) * D
    a = torch.randn(n, C + pad, device="cuda").bfloat16().requires_grad_()  # pad: rows further apart than they are long
    ws = [torch.nn.Parameter((torch.rand(D, device="cuda") + 0.5).bfloat16()) for _ in range(2)] if norm else [None, None]
    for w in ws if norm else []:
        w.main_grad = torch.ones(D, device="cuda")
    ang = torch.rand(n, D // 2, device="cuda").repeat(1, 2) * 6
    cos, sin = ang.cos().bfloat16(), ang.sin().bfloat16()
    q, k, v = qk_norm_rope(a[:, :C], ws[0], ws[1], cos, sin, Hq, Hkv, D, 1e-6)
    a64 = a.detach().double().requires_grad_()
    w64 = [w.detach().double().requires_grad_() for w in ws] if norm else ws

    def rotated(t, w):
        if w is not None:
            t = t * (t.pow(2).mean(-1, keepdim=True) + 1e-6).rsqrt() * w
        return t * cos.double()[:, None] + torch.cat([-t[..., D // 2:], t[..., :D // 2]], -1) * sin.double()[:, None]

    wants = [rotated(a64[:, :Hq * D].view(n, Hq, D), w64[0]), rotated(a64[:, Hq * D:(Hq + Hkv) * D].view(n, Hkv, D), w64[1]),
             a64[:, (Hq + Hkv) * D:C].view(n, Hkv, D)]
    outs = [q, k, v]
    if not with_dv:
        outs, wants = outs[:2], wants[:2]
    ds = [torch.randn_like(t) for t in outs]
    torch.autograd.backward(outs, ds)
    torch.autograd.backward(wants, [d.double() for d in ds])
    assert ((a.grad.double() - a64.grad).abs() <= BF16_MAX * a64.grad.abs() + 1e-5 * a64.grad.abs().max()).all()
    for w, d in zip(ws, w64) if norm else []:
        assert _rel(w.main_grad - 1, d.grad) < 1e-5


def test_updates_and_bounds_without_elements():
    from pithtrain_b200.modules.optimizer import Muon

    w = torch.empty(0, 8, 16, device="cuda", dtype=torch.bfloat16)
    Muon([torch.nn.Parameter(w)])._update_chunk(w, w.float(), w.float(), 0.95, 0.1, 0.0)
    cu = torch.zeros(2, dtype=torch.int32, device="cuda")
    assert N.row_lower_bounds(1, 0, 0, None, cu, cu.device).numel() == 0
    with pytest.raises(RuntimeError):
        N.row_lower_bounds(1, 4, 0, None, torch.zeros(2, 2, dtype=torch.int32, device="cuda"), cu.device)


@pytest.mark.parametrize("docs", [[0, 1], [0, 7, 7, 8, 300], [0, 128, 256, 257], [0, 0, 5, 5], [3, 10, 700]])
def test_packed_positions(docs):
    """Against the tensor-op form on the CPU: empty documents, boundaries that do not start at 0."""
    from pithtrain_b200.models.common import packed_positions

    for dtype in (torch.int32, torch.int64):
        cu = torch.tensor(docs, dtype=dtype)
        S = docs[-1] - docs[0]
        got = packed_positions(S, cu.cuda())
        assert got.dtype == torch.int64 and torch.equal(got.cpu(), packed_positions(S, cu))


def test_tensors_of_another_device_take_the_tensor_operations(monkeypatch):
    """Launches go to the current device: with the tensors on another one, no kernel may be handed their memory."""
    from pithtrain_b200.models.common import packed_positions
    from pithtrain_b200.modules.load_balance import force_balance
    from pithtrain_b200.ops.router import router_replayed

    cu, dev = torch.tensor([0, 3, 3, 9], dtype=torch.int32, device="cuda"), torch.device("cuda", torch.cuda.current_device())
    picks, logits = torch.zeros(9, 2, dtype=torch.int32, device="cuda"), torch.randn(9, 8, device="cuda")
    calls = [lambda: (packed_positions(9, cu),), lambda: (N.row_lower_bounds(1, 9, 0, 4, cu, dev),), lambda: (force_balance(8)(picks),),
             lambda: router_replayed(logits, 2, force_balance(8), True)]
    want = [c() for c in calls]

    def no_launch(rc, what):
        raise AssertionError(what)

    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 99)
    monkeypatch.setattr(_native, "check", no_launch)
    for c, w in zip(calls, want):
        for a, b in zip(c(), w):
            torch.testing.assert_close(a, b, rtol=1e-6, atol=0)


def test_layer_passes_refuse_inputs_on_another_device():
    """Weights, gates and rotary tables elsewhere, or a weight that the general form would repeat over the channels, do not
    reach the kernels as addresses."""
    from pithtrain_b200.ops import gated_attn as GA, gdn_mix, mla

    mk = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    x, w = mk(4, 128), mk(128)
    assert gdn_mix.gated_norm_supported(x, x, w)
    for z, u in ((x.cpu(), w), (x, w.cpu()), (x, w[:1])):
        assert not gdn_mix.gated_norm_supported(x, z, u)
    taps = mk(3 * 128, 1, 4)
    assert gdn_mix.conv_supported(mk(1, 5, 384), taps, 1, 1, 128, 128) and not gdn_mix.conv_supported(mk(1, 5, 384), taps.cpu(), 1, 1, 128, 128)
    qkv, c = mk(4, 512), mk(4, 32)
    assert GA.gated_attn_supported(qkv, w, w, 32, 1, 1, 128)
    assert not GA.gated_attn_supported(qkv, w, w.cpu(), 32, 1, 1, 128)
    args = (mk(4, 192), mk(4, 64), mk(4, 256), mk(4, 64), mk(4, 64), torch.arange(4, device="cuda"))
    for i in range(2):
        with pytest.raises(RuntimeError):
            GA.gated_attn_pre(qkv, w, w, *(t.cpu() if i == j else t for j, t in enumerate((c, c))), 1, 1, 128, 1e-6)
    for i in range(1, 6):
        with pytest.raises(RuntimeError):
            mla.mla_assemble(*(t.cpu() if i == j else t for j, t in enumerate(args)), 4, 1, 128, 64, 128)


@pytest.mark.parametrize("positions", [None, [0, 1, 7, 3], [2, -8, 0, -1], [2, -9, 0, 1]])
def test_mla_positions_outside_the_rotary_tables(positions):
    """Negative positions count from the end of the tables, as an index does; one outside them is never read, shows as NaN both
    ways and is reported."""
    from pithtrain_b200.ops import mla

    torch.manual_seed(4)
    n, rows = 4, 3 if positions is None else 8
    bad = next((i for i, x in enumerate(positions or range(n)) if not -rows <= x < rows), None)
    q, kp, kv = (torch.randn(n, c, device="cuda").bfloat16().requires_grad_() for c in (2 * 32, 16, 2 * 32))
    cos, sin = (torch.rand(rows, 16, device="cuda").bfloat16() for _ in range(2))
    pos = None if positions is None else torch.tensor(positions, device="cuda")
    out = mla.mla_assemble(q, kp, kv, cos, sin, pos, n, 2, 16, 16, 16)
    grads = torch.autograd.grad(out, (q, kp, kv), [torch.ones_like(t) for t in out])
    if bad is None:
        _native.check_status()
        same = mla.mla_assemble(q, kp, kv, cos, sin, pos % rows, n, 2, 16, 16, 16)
        assert all(torch.equal(a, b) for a, b in zip(out, same))
    else:
        with pytest.raises(_native.KernelStatusError):
            _native.check_status()
    for t, part in ((out[0], slice(16, None)), (out[1], slice(16, None)), (grads[0].view(n, 2, 32), slice(16, None)), (grads[1][:, None], slice(None))):
        assert [bool(x) for x in t[..., part].isnan().all(-1).all(-1)] == [i == bad for i in range(n)]
    assert torch.isfinite(out[2]).all() and torch.isfinite(grads[2]).all()


@pytest.mark.parametrize("Hkv,launches", [(4, 4), (2, 6)])
def test_launch_count_of_the_split_backward(Hkv, launches):
    """The row sums, dQ, dK and dV, and the sums of dK and dV over a group of heads where there are groups."""
    q, do = (torch.randn(1, 5, 4, 64, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(1, 5, Hkv, 64, device="cuda").bfloat16() for _ in range(2))
    out, lse = N.forward(q, k, v, 0.125, True, 0, None, None)
    before = _native.LAUNCHES
    N.backward_split(do, q, k, v, out, lse, 0.125, True, 0, None)
    assert _native.LAUNCHES - before == launches


def test_layer_passes_refuse_other_shapes():
    """What a reshape or a broadcast of the tensor operations refused: rows or widths that the kernels would read past."""
    from pithtrain_b200.ops import gated_attn as GA, gdn_mix, mla

    mk = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    taps, w, qkv, c = mk(3 * 128, 1, 4), mk(128), mk(4, 512), mk(4, 32)
    assert gdn_mix.conv_supported(mk(1, 5, 384), taps, 1, 1, 128, 128) and not gdn_mix.conv_supported(mk(1, 5, 256), taps, 1, 1, 128, 128)
    for bad in ((c[:3], c[:3]), (c, c[:, :16]), (c.float(), c.float())):
        with pytest.raises(RuntimeError):
            GA.gated_attn_pre(qkv, w, w, *bad, 1, 1, 128, 1e-6)
    o = mk(4, 1, 128)
    with pytest.raises(RuntimeError):
        GA.gated_attn_post(o, GA.gated_attn_pre(qkv, w, w, c, c, 1, 1, 128, 1e-6)[3][:3])
    args = [mk(4, 192), mk(4, 64), mk(4, 256), mk(4, 64), mk(4, 64), torch.arange(4, device="cuda")]
    mla.mla_assemble(*args, 4, 1, 128, 64, 128)
    for i in range(6):
        for bad in (args[i][:3], args[i][..., :-1], args[i].double()) if i < 5 else (args[i][:3],):
            if i in (3, 4) and bad.shape == (3, 64):
                continue  # shorter tables: checked position by position
            with pytest.raises(RuntimeError):
                mla.mla_assemble(*(bad if i == j else t for j, t in enumerate(args)), 4, 1, 128, 64, 128)


# ------------------------------------------------------------------------------------------------
# operators with their host side in C++
# ------------------------------------------------------------------------------------------------
def _host_operators():
    """(name, function of its differentiable inputs, inputs): outputs as a tuple of differentiable tensors."""
    from pithtrain_b200.ops.attention import attention
    from pithtrain_b200.ops.linear import linear
    from pithtrain_b200.ops.moe import ExpertWeights, moe_experts
    from pithtrain_b200.ops.norm import rmsnorm
    from pithtrain_b200.ops.rope import qk_norm_rope
    from pithtrain_b200.ops.router import router_topk

    torch.manual_seed(21)
    mk = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    w, nw, hw = torch.nn.Parameter(mk(64, 128)), torch.nn.Parameter(mk(128)), torch.nn.Parameter(mk(64))
    cos, sin = mk(16, 64), mk(16, 64)
    w1, w2 = mk(4, 128, 64), mk(4, 64, 64)
    ew = ExpertWeights(w1, w2, lambda: torch.zeros(4, 128, 64, device="cuda"), lambda: torch.zeros(4, 64, 64, device="cuda"))
    eids = torch.randint(0, 4, (9, 2), dtype=torch.int32, device="cuda")
    return [
        ("linear", lambda x: (linear(x, w),), (mk(9, 128),)),
        ("rmsnorm", lambda x, r: rmsnorm(x, nw, 1e-6, r), (mk(9, 128), mk(9, 128))),
        ("rope", lambda x: qk_norm_rope(x, hw, hw, cos, sin, 2, 1, 64, S=9), (mk(9, 256),)),
        ("attention", lambda q, k, v: (attention(q, k, v),), (mk(1, 9, 2, 64), mk(1, 9, 1, 64), mk(1, 9, 1, 64))),
        ("router", lambda x: router_topk(x, 2, "softmax_topk", True)[::2], (mk(9, 16).float(),)),
        ("experts", lambda x, p: (moe_experts(x, p, eids, ew),), (mk(9, 64), torch.rand(9, 2, device="cuda"))),
    ]


@pytest.mark.parametrize("name", ["linear", "rmsnorm", "rope", "attention", "router", "experts"])
def test_host_operators_in_autograd(name):
    """Each output alone, strided and misaligned inputs and gradients, saved-tensor hooks, a changed input and transforms: as for an
    operator written in Python."""
    fn, inputs = next((f, i) for n, f, i in _host_operators() if n == name)
    leaves = [t.clone().requires_grad_() for t in inputs]
    outs = fn(*leaves)
    grads = [torch.randn(o.shape, device="cuda").to(o.dtype) for o in outs]
    want = torch.autograd.grad(outs, leaves, grads, retain_graph=True, allow_unused=True)
    # one output at a time; gradients are linear in them up to the rounding of each pass
    total = None
    for o, g in zip(outs, grads):
        part = [torch.zeros_like(t) if p is None else p for p, t in zip(torch.autograd.grad(o, leaves, g, retain_graph=True, allow_unused=True), leaves)]
        total = part if total is None else [a.float() + b.float() for a, b in zip(total, part)]
    for a, b in zip(total, want):
        assert float((a.float() - b.float()).norm()) <= 4 * BF16_NORM * float(b.float().norm()) + 1e-6

    def elsewhere(t):  # the same values, every other row (token) of a larger tensor that starts off a 16-byte boundary
        rows = 1 if t.dim() == 4 else 0
        shape = [2 * n if i == rows else n for i, n in enumerate(t.shape)]
        big = torch.zeros(1 + 2 * t.numel(), dtype=t.dtype, device="cuda")[1:].view(shape)
        part = big[:, ::2] if rows else big[::2]
        part.copy_(t)
        return part

    moved = [elsewhere(t.detach()).requires_grad_() for t in leaves]
    got_outs = fn(*moved)
    got = torch.autograd.grad(got_outs, moved, [elsewhere(g) for g in grads], allow_unused=True)
    for a, b in zip((*got_outs, *got), (*outs, *want)):
        torch.testing.assert_close(a, b, rtol=0, atol=0 if name != "attention" else 2e-2)  # its fp32 sums come by atomics
    saved = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (saved.append(1), t)[1], lambda t: t):
        hooked = fn(*leaves)
    for a, b in zip(torch.autograd.grad(hooked, leaves, grads, allow_unused=True), want):
        torch.testing.assert_close(a, b, rtol=0, atol=0 if name != "attention" else 2e-2)
    assert saved
    with torch.no_grad():
        assert not any(o.requires_grad for o in fn(*leaves))
    if name != "router":  # keeps only what it computed
        mine = [t.clone().requires_grad_() for t in inputs]
        temp = [t * 1 for t in mine]
        outs = fn(*temp)
        with torch.no_grad():
            temp[0 if name != "rmsnorm" else 1].add_(1)
        if name != "rmsnorm":  # with a residual it keeps their sum
            with pytest.raises(RuntimeError, match="modified by an inplace operation"):
                torch.autograd.grad(outs, mine, grads, allow_unused=True)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda *a: fn(*a))(*[torch.stack([t, t]) for t in inputs])
    with pytest.raises(RuntimeError):
        torch.func.jvp(lambda *a: fn(*a), tuple(inputs), tuple(torch.ones_like(t) for t in inputs))
    _native.check_status()


@pytest.mark.filterwarnings("ignore::DeprecationWarning", "ignore::torch.jit.TracerWarning")
@pytest.mark.parametrize("name", ["linear", "rmsnorm", "rope", "router", "router after top k", "experts"])
def test_host_operators_in_a_trace(name):
    """``torch.jit.trace`` records each operator as a call: other inputs, of other numbers of rows too, give the operator's outputs and
    gradients, not unwritten memory."""
    from pithtrain_b200.ops.linear import linear
    from pithtrain_b200.ops.moe import ExpertWeights, moe_experts
    from pithtrain_b200.ops.norm import rmsnorm
    from pithtrain_b200.ops.rope import qk_norm_rope
    from pithtrain_b200.ops.router import router_topk

    torch.manual_seed(27)
    mk = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    w, nw, hw, w1, w2 = mk(64, 128), mk(128), mk(64), mk(4, 128, 64), mk(4, 64, 64)  # constants of the trace
    for t in (w, nw, hw):
        t.main_grad = torch.zeros(t.shape, device="cuda")
    cos, sin = mk(32, 64), mk(32, 64)
    ew = ExpertWeights(w1, w2, lambda: torch.zeros(4, 128, 64, device="cuda"), lambda: torch.zeros(4, 64, 64, device="cuda"))
    picks = lambda n: torch.randint(0, 4, (n, 2), dtype=torch.int32, device="cuda")  # noqa: E731
    fn, inputs = {
        "linear": (lambda x: linear(x, w), lambda n: [mk(n, 128)]),
        "rmsnorm": (lambda x, r: rmsnorm(x, nw, 1e-6, r), lambda n: [mk(n, 128), mk(n, 128)]),
        "rope": (lambda x: qk_norm_rope(x, hw, hw, cos, sin, 2, 1, 64, S=32), lambda n: [mk(n, 256)]),
        "router": (lambda x: router_topk(x, 2, "softmax_topk", True), lambda n: [mk(n, 16).float()]),
        "router after top k": (lambda x: router_topk(x, 2, "topk_softmax")[:2], lambda n: [mk(n, 16).float()]),
        "experts": (lambda x, p, e: moe_experts(x, p, e, ew), lambda n: [mk(n, 64), torch.rand(n, 2, device="cuda"), picks(n)]),
    }[name]
    for grad in (False, True):
        with torch.set_grad_enabled(grad):
            example = lambda n: tuple(t.requires_grad_(grad and t.is_floating_point()) for t in inputs(n))  # noqa: E731
            traced = torch.jit.trace(fn, example(9), check_trace=False)
            for n in (9, 30, 1):
                args = example(n)
                leaves = [t for t in args if t.requires_grad]
                want, got = ((o,) if isinstance(o, torch.Tensor) else o for o in (fn(*args), traced(*args)))
                assert all(torch.equal(a, b) for a, b in zip(got, want))
                if grad:
                    dy = [torch.randn_like(o) if o.is_floating_point() else None for o in want]
                    grads = [torch.autograd.grad([o for o in outs if o.requires_grad], leaves, [d for o, d in zip(outs, dy) if o.requires_grad], retain_graph=True)
                             for outs in (want, got)]
                    assert all(torch.equal(a, b) for a, b in zip(*grads))
    _native.check_status()


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("hooks", ["identity", "copy", "memory trace", "checkpoint"])
def test_weight_gradients_under_saved_tensor_hooks(hooks, flat):
    """Hooks hand other tensors back than the parameters; the gradients reach the parameters all the same, and are the same."""
    from contextlib import nullcontext

    from torch.utils.checkpoint import checkpoint

    from pithtrain_b200.ops.linear import linear
    from pithtrain_b200.ops.norm import rmsnorm
    from pithtrain_b200.ops.rope import qk_norm_rope
    from pithtrain_b200.tools.memory_trace import SavedTensorBytes

    torch.manual_seed(25)
    mk = lambda *s: torch.randn(*s, device="cuda").bfloat16()  # noqa: E731
    start, cos, sin = [mk(*s) for s in ((128,), (128,), (256, 128), (64,), (64,))], mk(9, 64), mk(9, 64)
    x, res, dy = mk(9, 128), mk(9, 128), [mk(9, n, 64) for n in (2, 1, 1)]
    context = {"identity": lambda: torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t), "memory trace": SavedTensorBytes,
               "copy": lambda: torch.autograd.graph.saved_tensors_hooks(lambda t: t.clone(), lambda t: t.clone())}

    def gradients(hooked):
        n1, n2, w, qw, kw = params = [torch.nn.Parameter(t.clone()) for t in start]
        if flat:
            for p in params:
                p.main_grad = torch.zeros(p.shape, device="cuda")

        def block(x, res):
            y, h = rmsnorm(rmsnorm(x, n1), n2, 1e-6, res)
            return qk_norm_rope(linear(y + h, w), qw, kw, cos, sin, 2, 1, 64, S=9)

        leaves = [t.clone().requires_grad_() for t in (x, res)]
        if hooked and hooks == "checkpoint":
            outs = checkpoint(block, *leaves, use_reentrant=False)
        else:
            with context[hooks]() if hooked else nullcontext():
                outs = block(*leaves)
        torch.autograd.backward(outs, dy)
        return [p.main_grad if flat else p.grad for p in params] + [t.grad for t in leaves]

    for want, got in zip(gradients(False), gradients(True)):
        assert want is not None and bool(want.any())
        assert got is not None and torch.equal(got, want)
    _native.check_status()


def test_expert_weights_are_not_saved():
    """What the expert block saves are activations: hooks (offloading, the memory trace) do not see its weights."""
    from pithtrain_b200.ops.moe import ExpertWeights, moe_experts

    torch.manual_seed(26)
    w1, w2 = (torch.nn.Parameter(torch.randn(s, device="cuda").bfloat16()) for s in ((4, 128, 64), (4, 64, 64)))
    g1, g2 = torch.zeros(w1.shape, device="cuda"), torch.zeros(w2.shape, device="cuda")
    ew = ExpertWeights(w1, w2, lambda: g1, lambda: g2)
    x, p = torch.randn(9, 64, device="cuda").bfloat16().requires_grad_(), torch.rand(9, 2, device="cuda")
    eids = torch.randint(0, 4, (9, 2), dtype=torch.int32, device="cuda")
    storages, weights = set(), {t.untyped_storage().data_ptr() for t in (w1, w2)}
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (storages.add(t.untyped_storage().data_ptr()), t)[1], lambda t: t):
        out = moe_experts(x, p, eids, ew)
    assert x.untyped_storage().data_ptr() in storages and not weights & storages
    out.backward(torch.ones_like(out))
    assert g1.any() and g2.any()


@pytest.mark.parametrize("bias", [False, True])
def test_host_linear_defers_and_finds_its_gradients(bias):
    """Weight gradients go to the W phase while it is on, to ``main_grad`` where a parameter has one and to ``.grad`` otherwise."""
    from pithtrain_b200.dualpipe.utils import WeightGradStore
    from pithtrain_b200.ops.linear import linear
    from pithtrain_b200.ops.norm import rmsnorm

    torch.manual_seed(22)
    x = torch.randn(24, 64, device="cuda").bfloat16().requires_grad_()
    for flat in (False, True):
        w, b = (torch.nn.Parameter(torch.randn(s, device="cuda").bfloat16()) for s in ((32, 64), (32,)))
        nw = torch.nn.Parameter(torch.randn(64, device="cuda").bfloat16())
        if flat:
            for p in (w, b, nw):
                p.main_grad = torch.zeros(p.shape, device="cuda")
        y = linear(rmsnorm(x, nw), w, b if bias else None)
        WeightGradStore.enabled = True
        try:
            y.backward(torch.ones_like(y))
        finally:
            WeightGradStore.enabled = False
        of = (lambda p: p.main_grad) if flat else (lambda p: p.grad)
        assert of(w) is None or not of(w).any()
        WeightGradStore.flush()
        WeightGradStore.pop()
        h = rmsnorm(x.detach(), nw.detach()).double()
        assert _rel(of(w), torch.ones(32, 24, device="cuda", dtype=torch.float64) @ h) <= BF16_NORM
        assert of(nw).any() and (not bias or _rel(of(b), torch.full((32,), 24.0, device="cuda", dtype=torch.float64)) == 0)
    _native.check_status()


@pytest.mark.parametrize("slots,E,valid", [(0, 4, None), (1, 1, None), (31, 33, None), (8191, 3, 5000), (8193, 256, None), (70001, 1024, 69000), (300000, 129, None), (64, 1025, None)])
def test_route_sort_runs_and_capacity(slots, E, valid):
    """At the edges of the warps' runs (32 slots and up) and of the experts a thread scans; slots without an expert; too few rows."""
    from pithtrain_b200.ops import moe as M

    torch.manual_seed(slots)
    eids = torch.randint(-1, E + 1, (slots,), dtype=torch.int32, device="cuda")
    if E > 2:
        eids[torch.rand(slots, device="cuda") < 0.5] = 1  # one expert takes most
    nv = None if valid is None else torch.tensor([valid], dtype=torch.int32, device="cuda")
    cap = M.sorted_capacity(slots, E)
    got = M.route_sort(eids, E, cap, nv)
    _native.check_status()
    want_in = eids.cpu().clone()
    if valid is not None:
        want_in[valid:] = -1
    for a, b in zip(got, M.route_sort_ref(want_in, E, cap)):
        assert torch.equal(a.cpu(), b)
    rows = int(got[0][-1])
    if rows and E <= 1024:
        offs, row_of_slot, slot_of_row = M.route_sort(eids, E, rows - 1, nv)
        with pytest.raises(_native.KernelStatusError):
            _native.check_status()
        assert torch.equal(offs, got[0]) and bool((row_of_slot == -1).all()) and bool((slot_of_row == -1).all())


@pytest.mark.parametrize("n,V", [(1, 1), (5, 7), (3, 8), (300, 2047), (300, 2048), (9, 2056), (300, 4096), (9, 4104), (9, 8192), (9, 8201), (300, 12288), (9, 12296),
                                 (300, 16384), (300, 16392), (9, 40003)])
def test_cross_entropy_rows(n, V):
    """One block size and one row length after the other, whole vectors and rests, masked columns (minus infinity), shifted rows."""
    from pithtrain_b200.ops.cross_entropy import cross_entropy

    torch.manual_seed(V)
    ld = (V + 7) // 8 * 8
    buf = (torch.randn(n, ld, device="cuda") * 3 + 40 * torch.randn(n, 1, device="cuda")).bfloat16()
    if V > 32:
        buf[:, : V // 3] = float("-inf")  # whole threads without a finite column
    labels = torch.randint(V // 3 if V > 32 else 0, V, (n,), device="cuda")
    labels[0] = V - 1
    if n > 2:
        labels[1] = -100
    want_in = buf[:, :V].double().requires_grad_()
    want = torch.nn.functional.cross_entropy(want_in, labels, ignore_index=-100, reduction="none")
    want.sum().backward()
    logits = buf[:, :V].detach().requires_grad_()
    got = cross_entropy(logits * 1.0 if ld == V else logits.as_strided((n, V), (ld, 1)), labels)
    got.backward()
    # the arguments of 2^x are rounded at |logit| log2(e) < 400, the sum of V terms in blocks, each loss of about |logit| once
    assert abs(float(got.detach().double() - want.detach().sum())) <= 2.0 ** -14 * float(want.detach().abs().sum()) + 2.0 ** -16 * n
    g, w = logits.grad.double(), want_in.grad
    assert ((g - w).abs() <= BF16_MAX * w.abs() + 2.0 ** -14 * (w.abs() + 2.0 ** -8)).all()
    assert (g[labels == -100] == 0).all()


@pytest.mark.parametrize("V", [5, 8, 1000, 2056, 4104, 9496, 12296, 16384, 16392, 40003])
def test_cross_entropy_of_masked_and_large_logits(V):
    """Masks of any size, the lowest bf16 value among them, over the leading columns, the rest or a whole row, and logits so large that
    their product with log2(e) is none or is rounded off by whole numbers."""
    from pithtrain_b200.ops.cross_entropy import cross_entropy

    torch.manual_seed(V)
    ld, lowest = (V + 7) // 8 * 8, torch.finfo(torch.bfloat16).min
    masks = [lowest, -2.4e38, -1e30, -1e9, -1e4, float("-inf")]
    rows, labels = [], []
    for fill in masks:
        for lo, hi in ((0, V // 2), (V // 2, V - 1), (0, V - 1)):  # leading columns, the following ones, all but the last
            row = torch.randn(ld).mul_(3)
            row[lo:hi] = fill
            rows.append(row)
            labels.append(V - 1)
    for fill in (*masks[:5], 1e9, 1e30, 3e38):
        rows.append(torch.full((ld,), fill))  # every column alike: the loss is log V
        labels.append(V // 3)
    for peak in (1e9, 1e30, 3e38):
        row = torch.randn(ld)
        row[V // 2] = peak
        rows.append(row)
        labels.append(V // 2)
    buf = torch.stack(rows).cuda().bfloat16()
    label = torch.tensor(labels, device="cuda")
    want_in = buf[:, :V].double().requires_grad_()
    want = torch.nn.functional.cross_entropy(want_in, label, reduction="none")
    want.sum().backward()
    for i in range(len(rows)):  # two of a row at a time: a loss that is wrong is not hidden by the others
        logits = buf[[i, i]].detach().requires_grad_()
        got = cross_entropy((logits * 1.0)[:, :V], label[[i, i]])
        got.backward()
        loss = 2 * float(want[i].detach())
        # as in the test above; differences of the logits are exact or off by 2^-24 of themselves
        assert abs(float(got.detach().double()) - loss) <= 2.0 ** -20 * (abs(loss) + 8), i
        g, w = logits.grad[:, :V].double(), want_in.grad[i]
        assert ((g - w).abs() <= BF16_MAX * w.abs() + 2.0 ** -14 * (w.abs() + 2.0 ** -8)).all(), i


@pytest.mark.parametrize("n,V,H", [(1, 1, 8), (0, 5, 64), (37, 3, 264), (700, 90, 2048), (5000, 4, 8)])
def test_embedding_gradient(n, V, H):
    """Rows of one id add up, onto what the buffer holds; strided and misaligned gradients; fp32 buffers and bf16 ones."""
    from pithtrain_b200.ops.embedding import embedding

    torch.manual_seed(n)
    ids = torch.randint(0, V, (n,), device="cuda")
    for dy in (torch.randn(n, H, device="cuda").bfloat16(), torch.randn(n * H + 1, device="cuda").bfloat16()[1:].view(n, H),
               torch.randn(n, 1, device="cuda").bfloat16().expand(n, H), torch.randn(H, n, device="cuda").bfloat16().t()):
        start = torch.randn(V, H, device="cuda")
        want = start.double().index_add(0, ids, dy.double())
        size = start.abs().double().index_add(0, ids, dy.abs().double())
        w = torch.nn.Parameter(torch.randn(V, H, device="cuda").bfloat16())
        w.main_grad = start.clone()
        embedding(ids, w).backward(dy)
        assert ((w.main_grad.double() - want).abs() <= 2.0 ** -24 * (n + 1) * size).all()  # n fp32 additions at most, in any order
    w = torch.nn.Parameter(torch.zeros(V, H, device="cuda").bfloat16())
    embedding(ids, w).backward(torch.ones(n, H, device="cuda").bfloat16())
    # a bf16 .grad: counts are whole numbers, exact up to 256
    assert torch.equal(w.grad[:, 0].float().clamp(max=256), torch.bincount(ids, minlength=V).float().clamp(max=256))
    _native.check_status()


@pytest.mark.parametrize("n,H", [(1, 8), (7, 264), (8, 256), (9, 64), (203, 520), (4099, 2048)])
def test_embedding_gradient_of_equal_neighbours(n, H):
    """Runs of one id within and across a warp's eight rows, ids outside the table among them (recorded, skipped, and no end of a run),
    a last warp of fewer rows."""
    torch.manual_seed(n)
    V = 5
    ids = torch.randint(0, V, (n,), device="cuda").repeat_interleave(torch.randint(1, 14, (n,), device="cuda"))[:n].contiguous()
    if n > 8:
        ids[torch.rand(n, device="cuda") < 0.1] = V  # outside
    dy, start = torch.randn(n, H, device="cuda").bfloat16(), torch.randn(V, H, device="cuda")
    grad = start.clone()
    _native.check(_native.lib().pt_embedding_bwd(dy.data_ptr(), ids.data_ptr(), grad.data_ptr(), n, H, V, _native.stream_ptr()), "pt_embedding_bwd")
    assert bool(_native.fetch_status()) == bool((ids == V).any())
    want, size, inside = start.double(), start.double().abs(), ids < V
    want.index_add_(0, ids[inside], dy[inside].double())
    size.index_add_(0, ids[inside], dy[inside].double().abs())
    assert ((grad.double() - want).abs() <= 2.0 ** -24 * (n + 1) * size).all()  # n fp32 additions at most, in any order


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (1, 5120, 2048), (3, 136, 72), (64, 128, 64), (64, 2048, 4096), (64, 9496, 520), (65, 264, 1032), (127, 2048, 512), (128, 648, 4096),
                                   (129, 128, 2048), (200, 2048, 4096), (300, 376, 1024), (1000, 128, 2048), (64, 20000, 128)])
def test_dense_few_rows(M, N, K):
    """Row counts up to a tile and past it, feature and reduction remainders, every split of the reduction from one CTA to eight; rows
    of a wider tensor; the same bits in every run."""
    from pithtrain_b200.ops import gemm as G

    torch.manual_seed(M + N + K)
    wide = torch.randn(M, K + 16, device="cuda").bfloat16()
    for x in (torch.randn(M, K, device="cuda").bfloat16(), wide[:, 8 : K + 8]):
        w = torch.randn(N, K, device="cuda").bfloat16()
        got = G.gemm_nt(x, w)
        want = x.double() @ w.double().t()
        size = x.double().abs() @ w.double().abs().t()
        # the tensor core cuts sums off at 24 bits or so, K / 16 times at most, then one bf16 rounding
        assert ((got.double() - want).abs() <= BF16_MAX * want.abs() + 2.0 ** -22 * (K // 16 + 9) * size).all()
        assert torch.equal(got, G.gemm_nt(x, w))
    _native.check_status()


@pytest.mark.parametrize("M,N,K", [(1024, 512, 4096), (1025, 512, 4096), (1152, 520, 4104), (1281, 512, 4096), (300, 584, 10944), (4616, 1032, 264)])
def test_dense_gradients_of_fewer_waves(M, N, K):
    """Just past a whole wave of 256-row tiles and beyond what 128-row tiles save: input gradients [M, K], weight gradients [M, K] of
    1024 rows and more."""
    from pithtrain_b200.ops import gemm as G

    torch.manual_seed(M)
    m = (M + 7) // 8 * 8  # rows of a weight: a multiple of 8
    for R in (N, 1024 + N):
        dy, w = torch.randn(M, R, device="cuda").bfloat16(), torch.randn(R, K, device="cuda").bfloat16()
        want, size = dy.double() @ w.double(), dy.double().abs() @ w.double().abs()
        slack = 2.0 ** -22 * (R // 16 + 9) * size  # the tensor core cuts sums off at 24 bits or so, R / 16 times at most
        assert ((G.gemm_nn(dy, w).double() - want).abs() <= BF16_MAX * want.abs() + slack).all()
        dyt = torch.zeros(R, m, device="cuda").bfloat16()
        dyt[:, :M] = dy.t()
        grad = G.gemm_tn(dyt, w, out=torch.zeros(m, K, device="cuda"), accumulate=True)
        assert ((grad[:M].double() - want).abs() <= slack).all() and not grad[M:].any()
    _native.check_status()


@pytest.mark.parametrize("extra", [False, True])
@pytest.mark.parametrize("n,H", [(1, 8), (591, 2048), (592, 2056), (593, 4096), (1185, 520), (1777, 6152), (3, 8192)])
def test_rmsnorm_backward_rows(n, H, extra):
    """One row a block, one more than the blocks, several rows each; every number of vectors a thread; with and without a residual."""
    from pithtrain_b200.ops.norm import rmsnorm

    torch.manual_seed(n)
    x = torch.randn(n, H, device="cuda").bfloat16().requires_grad_()
    res = torch.randn(n, H, device="cuda").bfloat16().requires_grad_() if extra else None
    w = torch.nn.Parameter(torch.randn(H, device="cuda").bfloat16())
    w.main_grad = torch.zeros(H, device="cuda")
    out = rmsnorm(x, w, 1e-6, res) if extra else rmsnorm(x, w, 1e-6)
    y, h = out if isinstance(out, tuple) else (out, None)
    dy, dh = torch.randn_like(y), torch.randn_like(y)
    torch.autograd.backward([y, h] if extra else [y], [dy, dh] if extra else [dy])
    hd = (h.detach() if extra else x.detach()).double()
    rstd = (hd.square().mean(-1, keepdim=True) + 1e-6).rsqrt()
    g = dy.double() * w.detach().double()
    dx = rstd * (g - hd * rstd * (g * hd * rstd).mean(-1, keepdim=True)) + (dh.double() if extra else 0)
    dw = (dy.double() * hd * rstd).sum(0)
    # fp32 terms of size rstd (|g| + |xhat| |dot|) and |dh|, one bf16 rounding; dw: n fp32 additions at most
    size = rstd * (g.abs() + (hd * rstd).abs() * (g * hd * rstd).abs().mean(-1, keepdim=True)) + (dh.double().abs() if extra else 0)
    assert ((x.grad.double() - dx).abs() <= BF16_MAX * dx.abs() + 2.0 ** -16 * size).all()
    assert ((w.main_grad.double() - dw).abs() <= 2.0 ** -24 * (n + 8) * (dy.double() * hd * rstd).abs().sum(0)).all()
