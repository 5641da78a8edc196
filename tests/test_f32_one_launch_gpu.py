"""float32 backward: dK/dV tiles and dQ tiles in one launch, of which there may be very different numbers."""

import pytest
import torch

import triton_sigmoid_b200 as m
from tests.gpu_util import launch_form, make_inputs
from triton_sigmoid_b200._cabi import FORM_F32_16, FORM_F32_64, FORM_F32_TC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("B,H,Tq,Tk,form", [(1, 3, 1, 70, FORM_F32_16), (1, 2, 130, 5, FORM_F32_16), (2, 3, 63, 65, FORM_F32_16), (80, 2, 64, 65, FORM_F32_64),
                                            (90, 2, 128, 17, FORM_F32_64), (2, 4, 16, 1000, FORM_F32_TC), (2, 4, 1000, 64, FORM_F32_TC), (3, 4, 513, 640, FORM_F32_TC)])
def test_against_64_bits(B, H, Tq, Tk, form, causal, D):
    """Bound: ten times the error of one sum of 1000 terms with roundings of 2^-24 that do not line up, 2^-24 sqrt(1000) = 1.9e-6; a tile that
    is left out, or taken twice, changes a gradient by more than 1e-2 of it."""
    assert launch_form(B, H, Tq, Tk, D, torch.float32, True, causal) == form
    q, k, v, do = make_inputs(B, Tq, Tk, H, D, torch.float32, std=0.5, seed=Tq + Tk)
    leaf = [t.requires_grad_() for t in (q, k, v)]
    full = [torch.full((B,), n, dtype=torch.int32, device="cuda") for n in (Tk, Tq)]
    got = torch.autograd.grad(m.sigmoid_attention_padded(*leaf, *full, is_causal=causal, sigmoid_bias=-1.0), leaf, do)
    qd, kd, vd, dd = (t.detach().double().transpose(1, 2) for t in (q, k, v, do))
    p = torch.sigmoid(qd @ kd.transpose(-1, -2) / D ** 0.5 - 1.0)
    if causal:
        p = p.tril()
    ds = p * (1 - p) * (dd @ vd.transpose(-1, -2)) / D ** 0.5
    for name, a, r in zip(("dq", "dk", "dv"), got, (ds @ kd, ds.transpose(-1, -2) @ qd, p.transpose(-1, -2) @ dd)):
        r = r.transpose(1, 2)
        assert ((a - r).norm() / r.norm()).item() <= 1.9e-5, name
