"""Rows of packed tensors that belong to no sequence are zero in every output, whatever the memory held before: in front of the
first sequence, behind the last one, and rows of a sequence beyond the given maximum."""

import pytest
import torch

import triton_sigmoid_b200 as sa
from tests.gpu_util import launch_form
from triton_sigmoid_b200._cabi import FORM_BWD, FORM_BWD_BY_HEAD

pytestmark = pytest.mark.gpu


def _poison(shape, dtype):
    """Memory of this size goes back to the allocator full of NaN, for the outputs to be made from."""
    keep = [torch.full(shape, float("nan"), dtype=dtype, device="cuda") for _ in range(4)]
    del keep


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("n,H,D,dtype,form", [
    (3, 2, 64, torch.bfloat16, FORM_BWD),
    (40, 8, 64, torch.float16, FORM_BWD),
    (40, 8, 128, torch.bfloat16, FORM_BWD),
    (40, 8, 24, torch.bfloat16, FORM_BWD),
    (260, 8, 64, torch.bfloat16, FORM_BWD_BY_HEAD),
    (6, 2, 64, torch.float32, None),
])
def test_rows_outside_the_sequences(n, H, D, dtype, form, split, monkeypatch):
    T, cut, front, behind = 300, 260, 37, 1000
    if split:
        monkeypatch.setenv("SIGATTN_B200_BWD_SPLIT", "1")
    g = torch.Generator().manual_seed(n)
    lens = torch.randint(T // 2, T + 1, (n,), generator=g)
    lens[0], lens[n // 2], lens[-1] = T, 0, T
    cu = torch.cat([torch.zeros(1, dtype=torch.long), lens.cumsum(0)]) + front
    rows = int(cu[-1]) + behind
    if form is not None:
        assert launch_form(n, H, cut, cut, D, dtype, True, packed_rows=rows) == form
    at = torch.arange(rows)
    seq = (torch.searchsorted(cu, at, right=True) - 1).clamp(0, n - 1)
    inside = ((at >= front) & (at < cu[-1]) & (at - cu[seq] < cut)).cuda()
    cu = cu.int().cuda()
    leaf = [(torch.randn(rows, H, D, device="cuda") * 0.5).to(dtype).requires_grad_() for _ in range(3)]
    do = torch.randn(rows, H, D, device="cuda").to(dtype)
    _poison((rows, H, D), dtype)
    out = sa.sigmoid_attention_varlen(*leaf, cu, cu, cut, cut)
    _poison((rows, H, D), dtype)
    for t in (out,) + torch.autograd.grad(out, leaf, do):
        assert (t[~inside] == 0).all() and t.isfinite().all()
        assert (t[inside] != 0).any(dim=-1).all()


def test_no_sequences_at_all():
    leaf = [torch.randn(500, 2, 64, device="cuda", dtype=torch.float16).requires_grad_() for _ in range(3)]
    cu = torch.zeros(1, dtype=torch.int32, device="cuda")
    _poison((500, 2, 64), torch.float16)
    out = sa.sigmoid_attention_varlen(*leaf, cu, cu, 64, 64)
    _poison((500, 2, 64), torch.float16)
    for t in (out,) + torch.autograd.grad(out, leaf, torch.ones_like(out)):
        assert (t == 0).all()


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1025, 5000])
@pytest.mark.parametrize("H,D", [(1, 64), (3, 40), (9, 128)])
def test_many_short_sequences(n, H, D):
    """Every warp of the kernel that zeroes the gaps searches for its part of the offsets, and many parts hold several gaps."""
    cut, front, behind = 24, 5, 4000 if n == 33 else 3
    g = torch.Generator().manual_seed(n)
    lens = torch.randint(0, 41, (n,), generator=g)
    lens[0] = 41
    cu = torch.cat([torch.zeros(1, dtype=torch.long), lens.cumsum(0)]) + front
    rows = int(cu[-1]) + behind
    at = torch.arange(rows)
    seq = (torch.searchsorted(cu, at, right=True) - 1).clamp(0, n - 1)
    inside = ((at >= front) & (at < cu[-1]) & (at - cu[seq] < cut)).cuda()
    cu = cu.int().cuda()
    leaf = [(torch.randn(rows, H, D, device="cuda") * 0.5).bfloat16().requires_grad_() for _ in range(3)]
    do = torch.randn(rows, H, D, device="cuda").bfloat16()
    _poison((rows, H, D), torch.bfloat16)
    out = sa.sigmoid_attention_varlen(*leaf, cu, cu, cut, cut)
    _poison((rows, H, D), torch.bfloat16)
    for t in (out,) + torch.autograd.grad(out, leaf, do):
        assert (t[~inside] == 0).all() and t.isfinite().all()
        assert (t[inside] != 0).any(dim=-1).all()


def test_debug_mode_poisons_packed_outputs_too(monkeypatch):
    """Outputs of packed calls are made from memory that nobody has cleared: a row that no kernel writes has to show."""
    monkeypatch.setenv("SIGATTN_B200_DEBUG", "1")
    leaf = [torch.randn(300, 2, 64, device="cuda", dtype=torch.float16).requires_grad_() for _ in range(3)]
    cu = torch.tensor([0, 100, 300], dtype=torch.int32, device="cuda")
    do = torch.randn(300, 2, 64, device="cuda", dtype=torch.float16)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as seen:
        out = sa.sigmoid_attention_varlen(*leaf, cu, cu, 200, 200)
        grads = torch.autograd.grad(out, leaf, do)
    assert sum(e.name == "aten::fill_" for e in seen.events()) == 4
    assert all(t.isfinite().all() and (t != 0).any(dim=-1).all() for t in (out,) + grads)


@pytest.mark.parametrize("dtype,H,n", [(torch.bfloat16, 4, 6), (torch.bfloat16, 8, 200), (torch.float32, 4, 6), (torch.float32, 1, 2)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("split", [False, True])
def test_queries_without_keys_and_keys_without_queries(split, D, dtype, H, n, monkeypatch):
    """Their rows belong to a sequence, so they are the attention kernels' to write: zeros."""
    if split:
        monkeypatch.setenv("SIGATTN_B200_BWD_SPLIT", "1")
    T = 300
    lq, lk = torch.full((n,), T), torch.full((n,), T)
    lq[::2] = torch.tensor([T, 0, 17]).repeat(n)[:len(lq[::2])]
    lk[1::2] = torch.tensor([0, 129, T]).repeat(n)[:len(lk[1::2])]
    cq, ck = (torch.cat([torch.zeros(1, dtype=torch.long), x.cumsum(0)]).int().cuda() for x in (lq, lk))
    alive = (lq > 0) & (lk > 0)
    rows_q, rows_k = (torch.repeat_interleave(alive, x).cuda() for x in (lq, lk))
    q, do = ((torch.randn(int(lq.sum()), H, D, device="cuda") * 0.5).to(dtype) for _ in range(2))
    k, v = ((torch.randn(int(lk.sum()), H, D, device="cuda") * 0.5).to(dtype) for _ in range(2))
    leaf = [t.requires_grad_() for t in (q, k, v)]
    _poison(q.shape, dtype)
    out = sa.sigmoid_attention_varlen(*leaf, cq, ck, T, T)
    _poison(q.shape, dtype), _poison(k.shape, dtype)
    for t, live in zip((out,) + torch.autograd.grad(out, leaf, do), (rows_q, rows_q, rows_k, rows_k)):
        assert (t[~live] == 0).all() and t.isfinite().all()
        assert (t[live] != 0).any(dim=-1).all()
