"""Biases on both sides of the line (-3) from which the 16-bit kernels leave out the test for logits far below zero, with scores
of which some, none or all are below it, against the oracle."""

import pytest
import torch

import triton_sigmoid_b200 as m
from tests.gpu_util import check_against_oracle, launch_form, make_inputs
from triton_sigmoid_b200._cabi import FORM_BWD, FORM_BWD_BY_HEAD

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("bias,shift", [(-2.9, 0.0), (-3.1, 0.0), (0.0, 0.0), (0.5, 0.0), (0.0, -6.0), (-2.9, -3.0), (-9.0, 6.0)])
def test_line(bias, shift, D, causal, dtype):
    """`shift` moves every score: the first column of q times that of k.  (No larger bias: dS = P (1 - P) dP comes from P in 16
    bits, whose rounding of up to 2^-9 in bf16 1 - P magnifies by P / (1 - P): 0.3 % at 0.5, 11 % at 4, in every form.)"""
    q, k, v, do = make_inputs(1, 385, 385, 2, D, dtype, std=0.5, seed=D)
    q[..., 0] = 1.0
    k[..., 0] = shift * D ** 0.5 / 8
    q[..., 0] *= 8.0
    for t in (q, k, v):
        t.requires_grad_()
    check_against_oracle(m.sigmoid_attention, q, k, v, do, dtype, is_causal=causal, sigmoid_bias=bias)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,T,form", [(1, 4, 200, FORM_BWD), (592, 2, 129, FORM_BWD_BY_HEAD)])
def test_padded_and_by_head(B, H, T, form, D):
    dtype = torch.bfloat16
    assert launch_form(B, H, T, T, D, dtype, True) == form
    lens = torch.randint(1, T + 1, (B,), generator=torch.Generator().manual_seed(T), dtype=torch.int32).cuda()
    valid = (torch.arange(T, device="cuda")[None] < lens[:, None])[..., None, None]
    q, k, v, do = make_inputs(B, T, T, H, D, dtype, std=0.5, seed=T)
    with torch.no_grad():
        for t in (q, k, v, do):
            t.masked_fill_(~valid, float("nan"))
    leaf = [t.requires_grad_() for t in (q, k, v)]
    out = m.sigmoid_attention_padded(*leaf, lens, lens, sigmoid_bias=0.5)
    grads = torch.autograd.grad(out, leaf, do)
    ref_in = [t.detach().float().masked_fill(~valid, 0.0).requires_grad_() for t in (q, k, v)]
    p = torch.sigmoid(torch.einsum("bqhd,bkhd->bhqk", ref_in[0], ref_in[1]) / D ** 0.5 + 0.5)
    p = p * valid[:, None, None, :, 0, 0]
    ref = torch.einsum("bhqk,bkhd->bqhd", p, ref_in[2]) * valid
    ref_g = torch.autograd.grad(ref, ref_in, do.float().masked_fill(~valid, 0.0))
    for a, r in zip((out,) + grads, (ref,) + ref_g):
        assert a.isfinite().all() and (a.masked_select(~valid) == 0).all()
        assert ((a.float() - r).norm() / r.norm()).item() <= 1e-2


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("every", [0, 700, 96, 40])
def test_scores_far_below_zero_without_a_bias(every, D, dtype):
    """Logits about -10 take the short series, whose leading term is exact, also where the scores make them: no common factor on the
    probabilities beyond what the 16-bit type leaves (the polynomial for all logits has 3.0e-4 in fp16 and 1.7e-3 in bf16 there;
    the series in 16 bits at most e^-10 = 4.5e-5, plus the mean of some 10^6 roundings).  `every`: that many keys apart one at a score
    of 0, so that tests for the series fail now and then."""
    B, T, H = 4, 1300, 8
    q, k, v, do = make_inputs(B, T, T, H, D, dtype, std=0.4, seed=D + every)
    q[..., 0] = 8.0
    k[..., 0] = -10.0 * D ** 0.5 / 8
    if every:
        k[:, 5::every, :, 0] = 0.0
    v += 1.0
    leaf = [t.requires_grad_() for t in (q, k, v)]
    out = m.sigmoid_attention(*leaf, sigmoid_bias=0.0)
    got = (out,) + torch.autograd.grad(out, leaf, do)
    qd, kd, vd, dd = (t.detach().double().transpose(1, 2) for t in (q, k, v, do))
    p = torch.sigmoid(qd @ kd.transpose(-1, -2) / D ** 0.5)
    ds = p * (1 - p) * (dd @ vd.transpose(-1, -2)) / D ** 0.5
    ref = [t.transpose(1, 2) for t in (p @ vd, ds @ kd, ds.transpose(-1, -2) @ qd, p.transpose(-1, -2) @ dd)]
    rel, factor = {torch.float16: (1e-3, 1.5e-4), torch.bfloat16: (6e-3, 6e-4)}[dtype]
    for name, a, r in zip(("o", "dq", "dk", "dv"), got, ref):
        a = a.double()
        assert ((a - r).norm() / r.norm()).item() <= rel, name
        if not every:
            assert abs((a * r).sum() / (r * r).sum() - 1).item() <= factor, name


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,T,form", [(4, 16, 1300, FORM_BWD), (74, 16, 260, FORM_BWD_BY_HEAD)])
def test_the_same_bits_each_time(B, H, T, form, D):
    """Work items with and without scores far below zero, which CTAs take in any order: O, dK and dV do not show it.  (dQ is a sum in
    any order in one form.)"""
    assert launch_form(B, H, T, T, D, torch.bfloat16, True) == form
    q, k, v, do = make_inputs(B, T, T, H, D, torch.bfloat16, std=0.5, seed=D)
    q[..., 0] = 8.0
    k[..., 0] = -torch.rand(B, 1, H, device="cuda") * 9.0 * D ** 0.5 / 8
    k[:, 7::90, :, 0] *= torch.rand(B, 1, H, device="cuda").bfloat16()
    leaf = [t.requires_grad_() for t in (q, k, v)]
    first = None
    for _ in range(30):
        out = m.sigmoid_attention(*leaf, sigmoid_bias=0.0)
        got = [out.detach(), *torch.autograd.grad(out, leaf, do)[1:]]
        first = first or got
        assert all(torch.equal(a, b) for a, b in zip(got, first))
