"""The two tile shapes of the float32 kernels (chosen by how many 64-row tiles there are) at the edges of their tiles,
against the float64 oracle with the gates of tests/test_f32_gpu.py."""

import pytest
import torch

import triton_sigmoid_b200 as sa
from tests.gpu_util import launch_form, make_inputs
from tests.test_f32_gpu import _check
from triton_sigmoid_b200._cabi import FORM_F32_16, FORM_F32_64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,T,form", [(1, 1, 15, FORM_F32_16), (1, 2, 17, FORM_F32_16), (1, 1, 81, FORM_F32_16),
                                        (1, 90, 63, FORM_F32_64), (40, 2, 64, FORM_F32_64), (1, 80, 65, FORM_F32_64),
                                        (5, 9, 129, FORM_F32_64)])
def test_tile_edges(B, H, T, form, D, causal):
    for backward in (False, True):
        assert launch_form(B, H, T, T, D, torch.float32, backward, causal) == form
    q, k, v, do = make_inputs(B, T, T, H, D, torch.float32, std=0.5, seed=T + D, requires_grad=True)
    lens = torch.randint(1, T + 1, (B,), generator=torch.Generator().manual_seed(T), dtype=torch.int32)
    lens[0] = T
    with torch.no_grad():  # the oracle multiplies masked zeros with the padding: finite, but nothing a result may hold
        for t in (q, k, v, do):
            for b in range(B):
                t[b, int(lens[b]):] = 1.0e3
    lens = lens.cuda()
    _check(q, k, v, do, lens_q=lens, lens_k=lens, is_causal=causal, score_mod=torch.randn(B, T, device="cuda") * 0.5)


@pytest.mark.parametrize("lo,hi", [(-20, -10), (-10, -4), (-4, 0), (0, 8)])
def test_sigmoid_is_as_accurate_as_the_plain_formula(lo, hi):
    """One key, one-hot: O is the sigmoid of the query's first column.  Its RMS relative error against float64 is no larger
    than that of 1 / (1 + exp(-x)) in float32."""
    T, H = 4096, 16
    x = torch.linspace(lo, hi, T * H + 2, device="cuda", dtype=torch.float64)[1:-1].float().reshape(T, H)
    q = torch.zeros(1, T, H, 64, device="cuda")
    q[0, :, :, 0] = x
    one = torch.zeros(1, 1, H, 64, device="cuda")
    one[..., 0] = 1.0
    out = sa.sigmoid_attention_padded(q, one, one, scale=1.0, sigmoid_bias=0.0)[0, :, :, 0]
    ref = 1.0 / (1.0 + torch.exp(-x.double()))
    rms = lambda y: ((y.double() - ref) / ref).square().mean().sqrt().item()  # noqa: E731
    assert rms(out) <= rms(1.0 / (1.0 + torch.exp(-x)))


@pytest.mark.parametrize("H", [1, 80])  # 16-row tiles, 64-row tiles
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_nonfinite_values_pass_through_probabilities_of_zero(bad, causal, H):
    """dS = P (1 - P) dP of a visible pair is 0 * NaN = NaN also where P has underflowed; of a masked pair it is 0."""
    T, j = 200, 70
    assert launch_form(1, H, T, T, 64, torch.float32, True, causal) == (FORM_F32_16 if H == 1 else FORM_F32_64)
    q, k, v, do = make_inputs(1, T, T, H, 64, torch.float32, std=0.5, seed=1)
    v[:, j] = bad
    do[..., 0] = 1.0  # so that dP is not finite whatever the signs of the other columns
    do[..., 1:] = 0.0
    leaf = [t.requires_grad_() for t in (q, k, v)]
    out = sa.sigmoid_attention(*leaf, is_causal=causal, sigmoid_bias=-1000.0)
    dq, dk, dv = torch.autograd.grad(out, leaf, do)
    sees = torch.arange(T, device="cuda") >= (j if causal else 0)  # queries that see key j
    assert dq[:, sees].isnan().all() and (dq[:, ~sees] == 0).all()
    at = torch.arange(T, device="cuda") == j
    assert dk[:, at].isnan().all() and (dk[:, ~at] == 0).all() and (dv == 0).all()
