"""The float32 kernels on the tensor cores at the edges of their tiles (128 stationary rows, 64 streamed ones), against the
float64 oracle with the gates of tests/test_f32_gpu.py."""

import math

import pytest
import torch

import triton_sigmoid_b200 as sa
from oracle import sigattn_oracle as orc
from tests.gpu_util import launch_form, make_inputs, rel_l2
from tests.test_f32_gpu import _check
from triton_sigmoid_b200._cabi import FORM_F32_TC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [20, 32, 64, 72, 96, 128])
@pytest.mark.parametrize("T", [256, 257, 319, 385])
def test_tile_edges(T, D, causal):
    B, H = 6, 4
    for backward in (False, True):
        assert launch_form(B, H, T, T, D, torch.float32, backward, causal) == FORM_F32_TC
    q, k, v, do = make_inputs(B, T, T, H, D, torch.float32, std=0.5, seed=T + D, requires_grad=True)
    lens = torch.tensor([T, 128, 129, 63, 1, 0], dtype=torch.int32)
    with torch.no_grad():  # the oracle multiplies masked zeros with the padding: finite, but nothing a result may hold
        for t in (q, k, v, do):
            for b in range(B):
                t[b, int(lens[b]):] = 1.0e3
    lens = lens.cuda()
    _check(q, k, v, do, lens_q=lens, lens_k=lens, is_causal=causal, score_mod=torch.randn(B, T, device="cuda") * 0.5)


@pytest.mark.parametrize("Tq,Tk", [(256, 1000), (700, 300)])
def test_packed_and_cross_lengths(Tq, Tk):
    """Packed sequences, queries and keys of different lengths, views of a wider tensor; and that a call gives the same bits
    each time."""
    H, D = 4, 64
    lq, lk = [Tq, 130, 1, 0, 64], [Tk, 65, 200, 128, 0]
    cq, ck = ([0] + torch.tensor(x).cumsum(0).tolist() for x in (lq, lk))
    g = torch.Generator(device="cuda").manual_seed(Tq)
    wide = [torch.randn(n, H, D + 32, device="cuda", generator=g) * 0.5 for n in (cq[-1], ck[-1], ck[-1])]
    q, k, v = (t[..., 16:16 + D].detach().requires_grad_() for t in wide)
    do = torch.randn(cq[-1], H, D, device="cuda", generator=g) * 0.5
    cu = [torch.tensor(c, dtype=torch.int32, device="cuda") for c in (cq, ck)]

    def call():
        out = sa.sigmoid_attention_varlen(q, k, v, *cu, Tq, Tk)
        return (out.detach(),) + torch.autograd.grad(out, (q, k, v), do)

    got = call()
    assert all(torch.equal(a, b) for a, b in zip(got, call()))
    for i in range(len(lq)):
        if not lq[i] or not lk[i]:
            continue
        sl = [t[None, a[i]:a[i + 1]].detach() for t, a in ((q, cq), (k, ck), (v, ck), (do, cq))]
        ref = (orc.sigattn_forward(*sl[:3], work=torch.float64),) + orc.sigattn_backward(*sl, work=torch.float64)
        for name, x, a, r in zip(("o", "dq", "dk", "dv"), got, (cq, cq, ck, ck), ref):
            assert rel_l2(x[a[i]:a[i + 1]].double().cpu(), r[0]) <= 1e-5, (i, name)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf"), 3.4e38])
def test_values_that_the_parts_cannot_carry(bad, causal, D):
    """Infinities, NaN and floats beyond the largest bf16 number reach the results as single precision has them."""
    T, j = 800, 64
    q, k, v, do = make_inputs(1, T, T, 2, D, torch.float32, std=0.5, seed=1)
    v[:, j, 0, 0] = bad   # head 0: the value of one key
    k[:, j, 1] = 0.0
    k[:, j, 1, 0] = bad   # head 1: the scores of one key (huge, of both signs)
    q[:, :, 1, 0] = 0.5 * torch.sign(q[:, :, 1, 0]) + q[:, :, 1, 0]
    out = sa.sigmoid_attention(q, k, v, is_causal=causal, sigmoid_bias=-1.0)
    with torch.no_grad():
        x = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double()) / D ** 0.5 - 1.0
        p = torch.sigmoid(x)
        if causal:
            p = p.masked_fill(torch.ones(T, T, device="cuda").triu(1).bool(), 0.0)
        w = v.double().clone()
        w[:, j, 0, 0] = 0.0
        ref = torch.einsum("bhqk,bkhd->bqhd", p, w)
        ref[:, :, 0, 0] += torch.where(p[:, 0, :, j] > 0, p[:, 0, :, j] * bad, 0.0)
    got = out.double()
    sees = slice(j if causal else 0, None)
    if bad != bad:
        assert got[:, sees, 0, 0].isnan().all() and got[:, sees, 1].isnan().all()
        got[:, sees, 0, 0] = ref[:, sees, 0, 0] = 0.0
        got[:, sees, 1] = ref[:, sees, 1] = 0.0
    inf = ref.isinf()
    assert torch.equal(got[inf], ref[inf])
    got[inf] = ref[inf] = 0.0
    assert got.isfinite().all()
    scale = ref.abs().amax(dim=(0, 1, 3), keepdim=True).clamp(min=1e-30) if bad != 3.4e38 else ref.abs().clamp(min=1.0)
    assert ((got - ref).abs() / scale).max().item() <= 1e-5


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_nonfinite_values_pass_through_probabilities_of_zero(bad, causal, D):
    """As in tests/test_f32_tiles_gpu.py: dS = P (1 - P) dP of a visible pair is NaN also where P has underflowed."""
    T, j = 2112, 70
    assert launch_form(1, 2, T, T, D, torch.float32, True, causal) == FORM_F32_TC
    q, k, v, do = make_inputs(1, T, T, 2, D, torch.float32, std=0.5, seed=1)
    v[:, j] = bad
    do[..., 0] = 1.0
    do[..., 1:] = 0.0
    leaf = [t.requires_grad_() for t in (q, k, v)]
    out = sa.sigmoid_attention(*leaf, is_causal=causal, sigmoid_bias=-1000.0)
    dq, dk, dv = torch.autograd.grad(out, leaf, do)
    sees = torch.arange(T, device="cuda") >= (j if causal else 0)
    assert dq[:, sees].isnan().all() and (dq[:, ~sees] == 0).all()
    at = torch.arange(T, device="cuda") == j
    assert dk[:, at].isnan().all() and (dk[:, ~at] == 0).all() and (dv == 0).all()


def _against_float64(q, k, v, do, bias, causal=False, scale=None, more=0.0, logits=True):
    """Relative errors (2-norm) of O, dQ, dK, dV at most 1e-6 - the six products leave some 4e-7 over 2048 terms, the FMA kernels up
    to 9e-7 - plus what the rounding of the logit costs (2^-24 of it, as a factor of the probability; `logits`), plus half a unit of the
    smallest float where the results are that small, plus `more`."""
    B, T, H, D = q.shape
    for backward in (False, True):
        assert launch_form(B, H, T, T, D, torch.float32, backward) == FORM_F32_TC
    scale = D ** -0.5 if scale is None else scale
    leaf = [t.requires_grad_() for t in (q, k, v)]
    out = sa.sigmoid_attention(*leaf, is_causal=causal, scale=scale, sigmoid_bias=bias)
    got = (out,) + torch.autograd.grad(out, leaf, do)
    qd, kd, vd, dd = (t.detach().double().transpose(1, 2) for t in (q, k, v, do))
    x = qd @ kd.transpose(-1, -2) * scale + bias
    p = torch.sigmoid(x)
    if causal:
        p = p.tril()
    ds = p * torch.sigmoid(-x) * (dd @ vd.transpose(-1, -2))
    ref = [t.transpose(1, 2) for t in (p @ vd, ds @ kd * scale, ds.transpose(-1, -2) @ qd * scale, p.transpose(-1, -2) @ dd)]
    rounding = 2.0 ** -24 * x.clamp(max=0.0).abs().max().item() if logits else 0.0
    for name, a, r in zip(("o", "dq", "dk", "dv"), got, ref):
        smallest = 2.0 ** -150 / r.square().mean().sqrt().item()
        assert rel_l2(a, r) <= 1e-6 + rounding + smallest + more, (name, rel_l2(a, r), rounding, smallest)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("which", ["q", "k", "v", "do"])
@pytest.mark.parametrize("size", [1e-30, 1e-33, 1e-35, 1e-37, 1e-38])
def test_small_values_keep_their_bits(size, which, D):
    """bf16 parts of a float below 1e-33 reach into bf16's subnormal numbers."""
    q, k, v, do = make_inputs(1, 520, 520, 8, D, torch.float32, std=0.5, seed=D)
    t = dict(q=q, k=k, v=v, do=do)[which]
    t *= size
    if which in "qk":  # (the other one's gradient is as large as the scale, and must stay a float)
        do *= 1e-3
    _against_float64(q, k, v, do, -math.log(520.0), scale=1.0 / size if which in "qk" else None)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("bias", [-50.0, -75.0, -84.0, -87.0, -90.0, -95.0, -100.0])
def test_probabilities_down_to_the_smallest_float(bias, D):
    q, k, v, do = make_inputs(1, 520, 520, 8, D, torch.float32, std=0.5, seed=D)
    _against_float64(q, k, v * 1e6, do * 1e6, bias)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("score", [-20.0, -60.0, -84.0, -87.0, -90.0, -95.0, -100.0])
def test_large_scores(score, D):
    """Every score is about that: one product of 64 or 128.  The tensor core cuts off its sum after each of the D / 16 steps,
    up to 2^-23 of it."""
    q, k, v, do = make_inputs(1, 520, 520, 8, D, torch.float32, std=0.5, seed=D)
    q[..., 0] = 8.0
    k[..., 0] = score * D ** 0.5 / 8
    _against_float64(q, k, v * 1e6, do * 1e6, 0.0, more=D / 16 * 2.0 ** -23 * abs(score))


@pytest.mark.parametrize("D", [64, 128])
def test_scores_beyond_the_scaled_range(D):
    """Sums that are floats, but not 2^32 times: 2e28, 2e29 and 4e29, which a small scale and a large bias make ordinary logits
    of (-231000, -83000 and 83000)."""
    q, k, v, do = make_inputs(1, 520, 520, 8, D, torch.float32, std=0.5, seed=D)
    q[..., 0] = 2.0e14
    k[..., 0] = torch.tensor([1.0e14, 1.0e15, 2.0e15], device="cuda").repeat(174)[:520][None, :, None]
    scale = 2.0 ** -80
    out = sa.sigmoid_attention(q, k, v, scale=scale, sigmoid_bias=-3.0e29 * scale)
    assert rel_l2(out, v[:, 2::3].double().sum(1, keepdim=True).expand_as(out)) <= 1e-6


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("std", [0.5, 1.0, 4.0])
@pytest.mark.parametrize("T", [520, 2048])
def test_all_six_products_count(T, std, D):
    """1e-6 (see _against_float64): without one of the three smallest products the errors are 2.5e-6 to 2e-5 at these inputs (a
    computation of the split products in 64 bits).  std 4: scores up to 80."""
    q, k, v, do = make_inputs(1, T, T, 8, D, torch.float32, std=std, seed=T + D)
    _against_float64(q, k, v, do, -math.log(T), logits=False)


@pytest.mark.parametrize("lo,hi", [(-80, -20), (-20, -10), (-10, -4), (-4, 0), (0, 8)])
@pytest.mark.parametrize("bias", [0.0, -7.3, -60.0])
def test_sigmoid_of_a_score(bias, lo, hi):
    """One of 64 keys with a value, one-hot: O is the sigmoid of the query's first column.  The exponent y = scale score log2(e) is rounded
    (2^-24 of it) and has a rounded factor (three roundings at most 2^-24 each), beyond a bias of -44 also the rest of the bias; ex2.approx
    has 2 units, rcp.approx 1, their arguments and e^-bias one each: 2^-23 a unit, and half of one for the smallest results."""
    T, H, scale = 4096, 16, 0.1
    f32 = lambda y: torch.tensor(y, dtype=torch.float32).item()  # noqa: E731
    s = torch.linspace((lo - bias) / scale, (hi - bias) / scale, T * H + 2, device="cuda", dtype=torch.float64)[1:-1].float().reshape(T, H)
    q = torch.zeros(1, T, H, 64, device="cuda")
    q[0, :, :, 0] = s
    one = torch.zeros(1, 64, H, 64, device="cuda")
    one[:, 9, :, 0] = 1.0
    assert launch_form(1, H, T, 64, 64, torch.float32, False) == FORM_F32_TC
    out = sa.sigmoid_attention_padded(q, one, one, scale=scale, sigmoid_bias=bias)[0, :, :, 0].double()
    x = s.double() * f32(scale)
    ref = torch.sigmoid(x + f32(bias))
    bound = 2.0 ** -24 * 4 * (x.abs() + max(0.0, -44.0 - bias)) + 5 * 2.0 ** -23 + 2.0 ** -150 / ref
    assert (((out - ref).abs() / ref) <= bound).all()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("where", ["k", "v", "do"])
def test_backward_of_values_that_the_parts_cannot_carry(where, causal, D):
    """One value of 1e34, which turns into NaN in the parts, in a column that the other operand has as 1e-34: the gradients are
    ordinary numbers, which only the repeat in single precision gives (every query tile sees key 64, every key tile query 790).
    Columns are compared one by one, with the gate of tests/test_f32_gpu.py."""
    B, T, H = 3, 800, 2
    assert launch_form(B, H, T, T, D, torch.float32, True, causal) == FORM_F32_TC
    q, k, v, do = make_inputs(B, T, T, H, D, torch.float32, std=0.5, seed=D)
    other = dict(k=q, v=do, do=v)[where]
    dict(k=k, v=v, do=do)[where][:, 790 if where == "do" else 64, :, 1] = 1.0e34
    other[..., 1] *= 1.0e-34
    leaf = [t.requires_grad_() for t in (q, k, v)]
    out = sa.sigmoid_attention(*leaf, is_causal=causal, sigmoid_bias=0.0)
    got = (out,) + torch.autograd.grad(out, leaf, do)
    qd, kd, vd, dd = (t.detach().double().transpose(1, 2) for t in (q, k, v, do))
    p = torch.sigmoid(qd @ kd.transpose(-1, -2) / D ** 0.5)
    if causal:
        p = p.tril()
    ds = p * (1 - p) * (dd @ vd.transpose(-1, -2)) / D ** 0.5
    for name, a, r in zip(("o", "dq", "dk", "dv"), got, (p @ vd, ds @ kd, ds.transpose(-1, -2) @ qd, p.transpose(-1, -2) @ dd)):
        assert a.isfinite().all(), name
        err = (a.transpose(1, 2).double() - r).norm(dim=2) / r.norm(dim=2)
        assert err.max().item() <= 1e-5, (name, err.max().item())
