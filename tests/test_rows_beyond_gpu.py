"""Rows beyond the valid ones: those of a tile that straddles a length inside the tensor are cleared, those beyond the tensor's end are never
read, whatever lies there in memory.  Held against the same call on compact tensors with zeros in the padding."""

import pytest
import torch

import triton_sigmoid_b200 as sa
from tests.gpu_util import rel_l2

pytestmark = pytest.mark.gpu


def _run(entry, q, k, v, do, lens, causal):
    leaf = [t.detach().requires_grad_() for t in (q, k, v)]
    if entry == "padded":
        out = sa.sigmoid_attention_padded(*leaf, lens, lens, is_causal=causal)
    elif entry == "varlen":
        out = sa.sigmoid_attention_varlen(*leaf, lens, lens, 128 * 3, 128 * 3, is_causal=causal)
    else:
        out = sa.sigmoid_attention(*leaf, is_causal=causal)
    return [out.detach(), *torch.autograd.grad(out, leaf, do)]


def _same(got, want):
    for name, a, b in zip(("o", "dq", "dk", "dv"), got, want):
        assert torch.isfinite(a).all(), name
        if name == "dq":  # fp32 terms in another order, then one rounding: at most neighbouring 16-bit values
            assert rel_l2(a, b) <= 2.0 ** -9
        else:
            assert torch.equal(a, b), name


@pytest.mark.parametrize("D", [64, 96])
@pytest.mark.parametrize("entry", ["dense", "padded"])
@pytest.mark.parametrize("B,T,causal", [(3, 127, False), (3, 129, True), (3, 300, False), (3, 255, True), (600, 130, False)])
def test_nan_behind_the_tensor_and_in_the_padding(B, T, causal, entry, D):
    H, g = 2, torch.Generator(device="cuda").manual_seed(T + D)
    clean = [torch.randn(B, T, H, D, device="cuda", generator=g).mul(0.5).to(torch.bfloat16) for _ in range(4)]
    # some sequences end with the tensor, some inside it, one by a single row
    lens = torch.tensor(([T, T - 1, 1] * B)[:B], dtype=torch.int32, device="cuda")
    pad = torch.arange(T, device="cuda")[None, :, None, None] >= lens[:, None, None, None]
    dirty = []
    for t in clean:
        big = torch.full((B, T + 150, H, D), float("nan"), device="cuda", dtype=t.dtype)
        big[:, :T] = t
        if entry == "padded":
            t.masked_fill_(pad, 0)
            big[:, :T].masked_fill_(pad, float("nan"))
        dirty.append(big[:, :T])
    _same(_run(entry, *dirty, lens, causal), _run(entry, *clean, lens, causal))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_neighbours_of_packed_sequences(D, causal):
    """What the sequences beside one hold, NaN included, is nothing to it: the first tiles of each are also its neighbour's last ones."""
    H, n = 2, [1, 127, 129, 384, 200, 128]
    g = torch.Generator(device="cuda").manual_seed(D)
    cu = torch.tensor([0, *n], device="cuda").cumsum(0).to(torch.int32)
    q, k, v, do = (torch.randn(sum(n), H, D, device="cuda", generator=g).mul(0.5).to(torch.float16) for _ in range(4))
    got = _run("varlen", q, k, v, do, cu, causal)
    for i in range(0, len(n), 2):
        lo, hi = int(cu[i]), int(cu[i + 1])
        odd = [t.clone() for t in (q, k, v, do)]
        for t in odd:
            t[:lo] = float("nan")
            t[hi:] = float("nan")
        part = _run("varlen", *odd, cu, causal)
        _same([t[lo:hi] for t in part], [t[lo:hi] for t in got])
