"""Padded and packed batches whose work is handed out by falling length, at the edges of the rule (as many batch elements as are
sorted, one more) and with equal, empty and full lengths, against float32 torch math."""

import pytest
import torch

import triton_sigmoid_b200 as m
from tests.gpu_util import GRAD_REL_L2, O_TOL, launch_form, make_inputs, rel_l2
from triton_sigmoid_b200._cabi import FORM_BWD, FORM_BWD_BY_HEAD

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("B,H,T,D,form", [(2, 40, 600, 64, FORM_BWD), (150, 1, 300, 128, FORM_BWD), (512, 1, 200, 64, FORM_BWD),
                                          (513, 1, 200, 64, FORM_BWD), (512, 3, 140, 64, FORM_BWD_BY_HEAD),
                                          (150, 8, 200, 128, FORM_BWD_BY_HEAD)])
def test_lengths_in_any_order(B, H, T, D, form, causal):
    dtype = torch.bfloat16
    assert launch_form(B, H, T, T, D, dtype, True, causal) == form
    lens = torch.randint(0, T + 1, (B,), generator=torch.Generator().manual_seed(B), dtype=torch.int32)
    lens[0], lens[-1] = 0, T
    lens[1:B // 2] = lens[1:B // 2] // 64 * 64  # many equal ones
    lens = lens.cuda()
    valid = torch.arange(T, device="cuda")[None] < lens[:, None]
    q, k, v, do = make_inputs(B, T, T, H, D, dtype, std=0.5, seed=T, requires_grad=True)
    ref_in = [t.detach().float().requires_grad_() for t in (q, k, v)]
    ref = m.sigmoid_attention_ref(*ref_in, seq_lens_k=lens, seq_lens_q=lens, causal=causal) * valid[:, :, None, None]
    ref_g = torch.autograd.grad(ref, ref_in, do.float() * valid[:, :, None, None])

    out = m.sigmoid_attention_padded(q, k, v, seq_lens_k=lens, seq_lens_q=lens, is_causal=causal)
    grads = torch.autograd.grad(out, (q, k, v), do)
    assert (out[~valid] == 0).all() and (out.float() - ref).abs().max().item() <= O_TOL[dtype]
    for g, r in zip(grads, ref_g):
        assert (g[~valid] == 0).all() and rel_l2(g, r) <= GRAD_REL_L2

    # the same sequences packed: the lengths come from the offsets
    cu = torch.cat([lens.new_zeros(1), lens.cumsum(0)]).int()
    packed = [t.detach()[valid].requires_grad_() for t in (q, k, v)]
    out_p = m.sigmoid_attention_varlen(*packed, cu, cu, T, T, is_causal=causal)
    assert (out_p.float() - ref[valid]).abs().max().item() <= O_TOL[dtype]
    for g, r in zip(torch.autograd.grad(out_p, packed, do[valid]), ref_g):
        assert rel_l2(g, r[valid]) <= GRAD_REL_L2


def test_queries_and_keys_of_different_lengths():
    B, H, Tq, Tk, D = 40, 4, 300, 500, 64
    g = torch.Generator().manual_seed(1)
    lq, lk = (torch.randint(1, n + 1, (B,), generator=g, dtype=torch.int32).cuda() for n in (Tq, Tk))
    q, k, v, do = make_inputs(B, Tq, Tk, H, D, torch.float16, std=0.5, seed=2, requires_grad=True)
    valid = torch.arange(Tq, device="cuda")[None] < lq[:, None]
    ref_in = [t.detach().float().requires_grad_() for t in (q, k, v)]
    ref = m.sigmoid_attention_ref(*ref_in, seq_lens_k=lk, seq_lens_q=lq) * valid[:, :, None, None]
    ref_g = torch.autograd.grad(ref, ref_in, do.float())
    out = m.sigmoid_attention_padded(q, k, v, seq_lens_k=lk, seq_lens_q=lq)
    assert (out.float() - ref).abs().max().item() <= O_TOL[torch.float16]
    for a, r in zip(torch.autograd.grad(out, (q, k, v), do), ref_g):
        assert rel_l2(a, r) <= GRAD_REL_L2
