"""float32 tensor-core kernels with a tile's jobs split over a cluster: parts of unequal size, parts without work, the split last wave of more
tiles, and tiles that the FMA code computes again."""

import pytest
import torch

import triton_sigmoid_b200 as m
from tests.gpu_util import launch_form, make_inputs
from triton_sigmoid_b200._cabi import FORM_F32_TC

pytestmark = pytest.mark.gpu


def _exact(q, k, v, do, lens_q, lens_k, causal, bias):
    q, k, v, do = (t.detach().double().transpose(1, 2) for t in (q, k, v, do))
    seen = (torch.arange(k.shape[2], device="cuda") < lens_k[:, None])[:, None, None, :] & (torch.arange(q.shape[2], device="cuda") < lens_q[:, None])[:, None, :, None]
    if causal:
        seen = seen & torch.ones_like(seen[..., :, :].expand(-1, -1, q.shape[2], k.shape[2]), dtype=torch.bool).tril()
    p = torch.sigmoid(q @ k.transpose(-1, -2) / q.shape[-1] ** 0.5 + bias) * seen
    ds = p * (1 - p) * (do @ v.transpose(-1, -2)) / q.shape[-1] ** 0.5
    return [t.transpose(1, 2) for t in (p @ v, ds @ k, ds.transpose(-1, -2) @ q, p.transpose(-1, -2) @ do)]


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("B,H,Tq,Tk,causal", [
    (1, 1, 1100, 900, False),   # 15 jobs in two parts
    (1, 1, 4200, 4200, True),   # parts of tiles near the diagonal's start have no work
    (3, 1, 520, 2100, False),   # a sequence without keys, one without queries
    (2, 10, 1024, 1024, False), # 160 tiles: 148, and 12 split
    (1, 2, 130, 8200, False),   # few queries: eight parts of the forward
])
def test_against_64_bits(B, H, Tq, Tk, causal, D):
    """Bound: ten times 2^-24 sqrt(4200), roundings of a sum that do not line up; a part left out changes results by more than 1e-2."""
    assert launch_form(B, H, Tq, Tk, D, torch.float32, False, causal) == FORM_F32_TC
    q, k, v, do = make_inputs(B, Tq, Tk, H, D, torch.float32, std=0.5, seed=Tq + Tk)
    lens_q = torch.full((B,), Tq, dtype=torch.int32, device="cuda")
    lens_k = torch.full((B,), Tk, dtype=torch.int32, device="cuda")
    if B > 2:
        lens_k[1], lens_q[2] = 0, 0
    leaf = [t.requires_grad_() for t in (q, k, v)]
    if B <= 2 and Tq == Tk:
        run = lambda: m.sigmoid_attention(*leaf, is_causal=causal, sigmoid_bias=-1.0)
    else:
        run = lambda: m.sigmoid_attention_padded(*leaf, lens_k, lens_q, is_causal=causal, sigmoid_bias=-1.0)
    out = run()
    got = (out,) + torch.autograd.grad(out, leaf, do)
    again = run()
    assert torch.equal(out, again) and all(torch.equal(a, b) for a, b in zip(got[1:], torch.autograd.grad(again, leaf, do)))
    for name, a, r in zip(("o", "dq", "dk", "dv"), got, _exact(q, k, v, do, lens_q, lens_k, causal, -1.0)):
        assert ((a - r).norm() / r.norm()).item() <= 3.9e-5, name


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("key", [5, 1500])  # in the first and in the last part
def test_nan_in_one_part(key, D):
    """A NaN in V reaches every output of its column and no other one; the tiles are computed again as a whole."""
    q, k, v, do = make_inputs(1, 1600, 1600, 1, D, torch.float32, std=0.5, seed=key)
    v[0, key, 0, 3] = float("nan")
    out = m.sigmoid_attention(q, k, v, sigmoid_bias=-1.0)
    full = torch.full((1,), 1600, device="cuda")
    ref = _exact(q, k, v, do, full, full, False, -1.0)[0]
    assert torch.equal(out.isnan(), ref.isnan()) and out.isnan().sum() == 1600
    keep = ~ref.isnan()
    assert ((out[keep] - ref[keep]).norm() / ref[keep].norm()).item() <= 2.4e-5
