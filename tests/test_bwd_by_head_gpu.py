"""Backward with whole (batch element, head) pairs per CTA (many short sequences), against the general form of the same
kernel on slices of the batch, which are too few pairs for it, and against the oracle for a few elements."""

import pytest
import torch

import triton_sigmoid_b200 as sa
from oracle import sigattn_oracle as orc
from tests.gpu_util import GRAD_REL_L2, launch_form, rel_l2
from triton_sigmoid_b200._cabi import FORM_BWD, FORM_BWD_BY_HEAD

pytestmark = pytest.mark.gpu


def _enough(B, H):
    """A batch of at least B elements whose (batch element, head) pairs are enough for the form: 8 per SM."""
    return max(B, -(-8 * torch.cuda.get_device_properties(0).multi_processor_count // H))


@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("B,H,Tq,Tk,causal", [
    (75, 16, 1, 1, False),
    (75, 16, 128, 128, False),    # one key tile: nothing is accumulated
    (75, 16, 130, 300, False),    # a query tile of two rows, ragged last key tile
    (40, 30, 300, 300, True),     # every query tile has another last key tile
    (75, 16, 400, 150, True),     # query tiles behind the last key tile
    (75, 16, 100, 400, True),     # key tiles that no query sees (D = 64: the general form's business, with one query tile)
    (75, 16, 200, 400, True),
    (112, 16, 100, 700, False),   # six key tiles, as 12 pairs per SM allow
])
def test_matches_the_general_form(B, H, Tq, Tk, causal, D):
    dtype = torch.bfloat16 if Tq % 2 else torch.float16
    B = _enough(B, H)
    g = torch.Generator(device="cuda").manual_seed(Tq + D)
    mk = lambda T: (torch.randn(B, T, H, D, device="cuda", generator=g) * 0.7).to(dtype)
    q, k, v, do = mk(Tq), mk(Tk), mk(Tk), mk(Tq)
    cpu = torch.Generator().manual_seed(Tk)
    lq = torch.randint(1, Tq + 1, (B,), generator=cpu, dtype=torch.int32)
    lk = torch.randint(1, Tk + 1, (B,), generator=cpu, dtype=torch.int32)
    lq[0], lk[0], lk[1], lq[2] = Tq, Tk, 0, 0
    for b in range(B):  # what lies in the padding must not matter
        q[b, int(lq[b]):] = float("nan")
        do[b, int(lq[b]):] = float("nan")
        k[b, int(lk[b]):] = float("nan")
        v[b, int(lk[b]):] = float("nan")
    lq, lk = lq.cuda(), lk.cuda()

    def grads(s):
        leaf = [t[s].detach().requires_grad_() for t in (q, k, v)]
        out = sa.sigmoid_attention_padded(*leaf, seq_lens_k=lk[s], seq_lens_q=lq[s], is_causal=causal, sigmoid_bias=-3.0)
        return torch.autograd.grad(out, leaf, do[s])

    step = 20
    assert launch_form(B, H, Tq, Tk, D, dtype, True, causal) == (FORM_BWD if (Tq, Tk, D) == (100, 400, 64) else FORM_BWD_BY_HEAD)
    assert launch_form(step, H, Tq, Tk, D, dtype, True, causal) == FORM_BWD
    whole = grads(slice(0, B))
    for b0 in range(0, B, step):
        part = grads(slice(b0, min(B, b0 + step)))
        for name, a, r in zip("qkv", whole, part):
            a = a[b0:b0 + step]
            assert torch.isfinite(a).all()
            if name == "q":  # the same fp32 terms in another order, then one rounding: at most neighbouring 16-bit values
                assert rel_l2(a, r) <= 2.0 ** -9
            else:
                assert torch.equal(a, r)
    sl = slice(0, 4)
    ref = orc.sigattn_backward(*[torch.nan_to_num(t[sl]) for t in (q, k, v, do)], seq_lens_k=lk[sl], seq_lens_q=lq[sl],
                               is_causal=causal, sigmoid_bias=-3.0)
    mq = torch.arange(Tq)[None, :] < lq[sl].cpu()[:, None]
    assert whole[0][sl].cpu()[~mq].abs().sum().item() == 0  # rows beyond the valid length
    for a, r in zip(whole, ref):
        assert rel_l2(a[sl].float().cpu(), r) <= GRAD_REL_L2


@pytest.mark.parametrize("causal", [False, True])
def test_packed(causal):
    H, D = 8, 64
    n = -(-_enough(160, H) // 40) * 40
    lens = torch.randint(0, 420, (n,), generator=torch.Generator().manual_seed(3))
    lens[0], lens[1] = 419, 0
    cu = torch.cat([torch.zeros(1, dtype=torch.long), lens.cumsum(0)]).to(device="cuda", dtype=torch.int32)
    g = torch.Generator(device="cuda").manual_seed(4)
    q, k, v, do = [torch.randn(int(lens.sum()), H, D, device="cuda", generator=g).bfloat16() for _ in range(4)]

    def grads(q, k, v, do, cu):
        leaf = [t.detach().requires_grad_() for t in (q, k, v)]
        out = sa.sigmoid_attention_varlen(*leaf, cu, cu, 419, 419, is_causal=causal)
        return torch.autograd.grad(out, leaf, do)

    assert launch_form(n, H, 419, 419, D, q.dtype, True, causal, packed_rows=len(q)) == FORM_BWD_BY_HEAD
    assert launch_form(40, H, 419, 419, D, q.dtype, True, causal, packed_rows=int(cu[40])) == FORM_BWD
    whole = grads(q, k, v, do, cu)
    for i in range(0, n, 40):
        s = slice(int(cu[i]), int(cu[i + 40]))
        part = grads(q[s], k[s], v[s], do[s], cu[i:i + 41] - cu[i])
        for name, a, r in zip("qkv", whole, part):
            if name == "q":
                assert rel_l2(a[s], r) <= 2.0 ** -9
            else:
                assert torch.equal(a[s], r)


def test_packed_batch_of_mostly_short_sequences():
    """Enough pairs, but few rows for the longest sequence (the accumulator of total_q rows has no room for a region of it
    per CTA): the general form, with the results of the sequences by themselves."""
    H, D = 1, 64
    n = _enough(1200, H)
    lens = [16] * n
    lens[7], lens[500] = 700, 411
    cu = torch.tensor([0] + lens).cumsum(0).to(device="cuda", dtype=torch.int32)
    g = torch.Generator(device="cuda").manual_seed(4)
    q, k, v, do = [torch.randn(sum(lens), H, D, device="cuda", generator=g).bfloat16() for _ in range(4)]
    assert launch_form(n, H, 700, 700, D, q.dtype, True, packed_rows=len(q)) == FORM_BWD
    leaf = [t.detach().requires_grad_() for t in (q, k, v)]
    got = torch.autograd.grad(sa.sigmoid_attention_varlen(*leaf, cu, cu, 700, 700), leaf, do)
    for i in (0, 6, 7, 8, 499, 500, n - 1):
        s = slice(int(cu[i]), int(cu[i + 1]))
        ref = orc.sigattn_backward(*[t[s][None] for t in (q, k, v, do)])
        for a, r in zip(got, ref):
            assert rel_l2(a[s].float().cpu(), r[0]) <= GRAD_REL_L2


@pytest.mark.parametrize("D", [8, 40, 64, 120])
@pytest.mark.parametrize("Tq,causal", [(130, False), (300, True)])
def test_per_key_terms_narrow_heads_and_fused_views(Tq, causal, D):
    H, step = 16, 20
    B = _enough(75, H)
    assert launch_form(B, H, Tq, Tq, D, torch.bfloat16, True, causal) == FORM_BWD_BY_HEAD
    g = torch.Generator(device="cuda").manual_seed(Tq + D)
    qkv = torch.randn(B, Tq, 3, H, D, device="cuda", generator=g).bfloat16()
    do = torch.randn(B, H, Tq, D, device="cuda", generator=g).bfloat16().transpose(1, 2)  # [B, Tq, H, D], heads outermost
    mod = torch.randn(B, Tq, device="cuda", generator=g)

    def grad(s):
        leaf = qkv[s].detach().requires_grad_()
        out = sa.sigmoid_attention(*leaf.unbind(2), is_causal=causal, score_mod=mod[s])
        return torch.autograd.grad(out, leaf, do[s])[0]

    whole = grad(slice(0, B))
    for b0 in range(0, B, step):
        part = grad(slice(b0, min(B, b0 + step)))
        a = whole[b0:b0 + step]
        assert rel_l2(a[:, :, 0], part[:, :, 0]) <= 2.0 ** -9  # dQ: the same fp32 terms in another order, then one rounding
        assert torch.equal(a[:, :, 1:], part[:, :, 1:])
    ref = orc.sigattn_backward(*qkv[:2].unbind(2), do[:2], is_causal=causal, score_mod=mod[:2])
    for i, r in enumerate(ref):
        assert rel_l2(whole[:2, :, i].float().cpu(), r) <= GRAD_REL_L2
