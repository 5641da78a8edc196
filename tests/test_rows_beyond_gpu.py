"""Rows beyond the valid ones: those of a tile that straddles a length inside the tensor are cleared, those beyond the tensor's end are never
read, whatever lies there in memory.  Held against the same call on compact tensors with zeros in the padding."""

import pytest
import torch

import triton_sigmoid_b200 as sa
from tests.gpu_util import GRAD_REL_L2, blockwise_fp32_reference, launch_form, rel_l2
from triton_sigmoid_b200 import _cabi

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[False, True], ids=["fused", "deterministic"])
def deterministic(request, monkeypatch):
    monkeypatch.setenv("SIGATTN_B200_BWD_SPLIT", str(int(request.param)))
    return request.param


def _run(entry, q, k, v, do, lens, causal):
    leaf = [t.detach().requires_grad_() for t in (q, k, v)]
    if entry == "padded":
        out = sa.sigmoid_attention_padded(*leaf, lens, lens, is_causal=causal)
    elif entry == "varlen":
        out = sa.sigmoid_attention_varlen(*leaf, lens, lens, 128 * 3, 128 * 3, is_causal=causal)
    else:
        out = sa.sigmoid_attention(*leaf, is_causal=causal)
    return [out.detach(), *torch.autograd.grad(out, leaf, do)]


# largest relative errors of the two polynomials between which a warp chooses, and two roundings of a probability
CHOICE = {torch.float16: 3.0e-4 + 3.1e-5 + 2.0 ** -11, torch.bfloat16: 1.74e-3 + 9.8e-4 + 2.0 ** -8}


def _same(got, want, deterministic):
    for name, a, b in zip(("o", "dq", "dk", "dv"), got, want):
        assert torch.isfinite(a).all(), name
        if name != "o" and deterministic:  # rows of its own tile beyond a length have a say in the polynomial that their warp takes
            assert rel_l2(a, b) <= CHOICE[a.dtype], name
        elif name == "dq":  # fp32 terms in another order, then one rounding: at most neighbouring 16-bit values
            assert rel_l2(a, b) <= 2.0 ** -9
        else:
            assert torch.equal(a, b), name


@pytest.mark.parametrize("D", [32, 64, 96])
@pytest.mark.parametrize("entry", ["dense", "padded"])
@pytest.mark.parametrize("B,T,causal", [(3, 127, False), (3, 129, True), (3, 300, False), (3, 255, True), (600, 130, False)])
def test_nan_behind_the_tensor_and_in_the_padding(B, T, causal, entry, D, deterministic):
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
    assert deterministic or launch_form(B, H, T, T, D, torch.bfloat16, True, causal) == (_cabi.FORM_BWD_BY_HEAD if B == 600 else _cabi.FORM_BWD)
    _same(_run(entry, *dirty, lens, causal), _run(entry, *clean, lens, causal), deterministic)


@pytest.mark.parametrize("D,dtype", [(32, torch.float16), (64, torch.bfloat16), (128, torch.bfloat16), (128, torch.float16)])
@pytest.mark.parametrize("bias", [None, 0.0])
@pytest.mark.parametrize("short", ["queries", "keys", "both", "keys, no lengths of queries"])
@pytest.mark.parametrize("Tq,Tk,causal", [(300, 200, False), (130, 390, False), (200, 333, True)])
def test_lengths_of_queries_and_keys(Tq, Tk, causal, short, bias, D, dtype, deterministic):
    """Queries that end with their tensor beside keys that do not, and the reverse: against the same call with zeros in the padding, and against
    plain arithmetic."""
    B, H, g = 3, 2, torch.Generator(device="cuda").manual_seed(Tq + D)
    lens_q = torch.tensor([Tq - 1, 1, Tq // 2] if short in ("queries", "both") else [Tq] * B, dtype=torch.int32, device="cuda")
    lens_k = torch.tensor([Tk - 1, Tk // 2, 1] if short != "queries" else [Tk] * B, dtype=torch.int32, device="cuda")
    clean, dirty = [], []
    for T, lens in ((Tq, lens_q), (Tk, lens_k), (Tk, lens_k), (Tq, lens_q)):
        pad = torch.arange(T, device="cuda")[None, :, None, None] >= lens[:, None, None, None]
        t = torch.randn(B, T, H, D, device="cuda", generator=g).mul(0.5).to(dtype).masked_fill_(pad, 0)
        big = torch.full((B, T + 150, H, D), float("nan"), device="cuda", dtype=dtype)
        big[:, :T] = t.masked_fill(pad, float("nan"))
        clean.append(t)
        dirty.append(big[:, :T])
    assert deterministic or launch_form(B, H, Tq, Tk, D, dtype, True, causal) == _cabi.FORM_BWD

    def run(q, k, v, do):
        leaf = [t.detach().requires_grad_() for t in (q, k, v)]
        out = sa.sigmoid_attention_padded(*leaf, lens_k, None if "no lengths" in short else lens_q, is_causal=causal, sigmoid_bias=bias)
        return [out.detach(), *torch.autograd.grad(out, leaf, do)]

    got = run(*dirty)
    _same(got, run(*clean), deterministic)
    b = None if bias is None else torch.zeros(B, device="cuda").view(B)
    for name, a, r in zip(("o", "dq", "dk", "dv"), got, blockwise_fp32_reference(*clean, lens_q, lens_k, causal, bias=b)):
        assert rel_l2(a, r) <= GRAD_REL_L2, name


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_neighbours_of_packed_sequences(D, causal, deterministic):
    """What the sequences beside one hold, NaN included, is nothing to it: the first tiles of each are also its neighbour's last ones."""
    H, n = 2, [1, 127, 129, 384, 200, 128]
    g = torch.Generator(device="cuda").manual_seed(D)
    cu = torch.tensor([0, *n], device="cuda").cumsum(0).to(torch.int32)
    q, k, v, do = (torch.randn(sum(n), H, D, device="cuda", generator=g).mul(0.5).to(torch.float16) for _ in range(4))
    assert deterministic or launch_form(len(n), H, 384, 384, D, torch.float16, True, causal, packed_rows=sum(n)) == _cabi.FORM_BWD
    got = _run("varlen", q, k, v, do, cu, causal)
    for i in range(0, len(n), 2):
        lo, hi = int(cu[i]), int(cu[i + 1])
        odd = [t.clone() for t in (q, k, v, do)]
        for t in odd:
            t[:lo] = float("nan")
            t[hi:] = float("nan")
        part = _run("varlen", *odd, cu, causal)
        _same([t[lo:hi] for t in part], [t[lo:hi] for t in got], deterministic)
