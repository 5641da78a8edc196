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
