"""Backward with whole (batch element, head) pairs per CTA (many short sequences), against the general form of the same
kernel on slices of the batch, which are too few pairs for it, and against the oracle for a few elements."""

import pytest
import torch

import triton_sigmoid_b200 as sa
from oracle import sigattn_oracle as orc
from tests.gpu_util import GRAD_REL_L2, rel_l2

pytestmark = pytest.mark.gpu


# (the pairs must be at least 8 per SM: 1184 on 148 SMs)
@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("B,H,Tq,Tk,causal", [
    (75, 16, 1, 1, False),
    (75, 16, 128, 128, False),    # one key tile: nothing is accumulated
    (75, 16, 130, 300, False),    # a query tile of two rows, ragged last key tile
    (40, 30, 300, 300, True),     # every query tile has another last key tile
    (75, 16, 400, 150, True),     # query tiles behind the last key tile
    (75, 16, 100, 400, True),     # key tiles that no query sees
])
def test_matches_the_general_form(B, H, Tq, Tk, causal, D):
    dtype = torch.bfloat16 if Tq % 2 else torch.float16
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

    whole = grads(slice(0, B))
    step = 20
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
    H, D, n = 8, 64, 160
    lens = torch.randint(0, 420, (n,), generator=torch.Generator().manual_seed(3))
    lens[0], lens[1] = 419, 0
    cu = torch.cat([torch.zeros(1, dtype=torch.long), lens.cumsum(0)]).to(device="cuda", dtype=torch.int32)
    g = torch.Generator(device="cuda").manual_seed(4)
    q, k, v, do = [torch.randn(int(lens.sum()), H, D, device="cuda", generator=g).bfloat16() for _ in range(4)]

    def grads(q, k, v, do, cu):
        leaf = [t.detach().requires_grad_() for t in (q, k, v)]
        out = sa.sigmoid_attention_varlen(*leaf, cu, cu, 419, 419, is_causal=causal)
        return torch.autograd.grad(out, leaf, do)

    whole = grads(q, k, v, do, cu)
    for i in range(0, n, 40):
        s = slice(int(cu[i]), int(cu[i + 40]))
        part = grads(q[s], k[s], v[s], do[s], cu[i:i + 41] - cu[i])
        for name, a, r in zip("qkv", whole, part):
            if name == "q":
                assert rel_l2(a[s], r) <= 2.0 ** -9
            else:
                assert torch.equal(a[s], r)
