"""The native eager path: inputs the kernels read in place (views of a fused projection) and inputs that have to be
copied first (misaligned, expanded) give the results of contiguous tensors; autograd's usual guarantees hold."""

import pytest
import torch

import triton_sigmoid_b200 as m

pytestmark = pytest.mark.gpu


def _views(kind, B, T, H, D, dtype):
    g = torch.Generator(device="cuda").manual_seed(7)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).to(dtype)  # noqa: E731
    if kind == "fused":            # [B, T, 3, H, D]
        return rand(B, T, 3, H, D).unbind(2)
    if kind == "head_major":       # [B, H, T, D] seen as [B, T, H, D]
        return [rand(B, H, T, D).transpose(1, 2) for _ in range(3)]
    if kind == "misaligned":       # rows that start off a 16-byte boundary
        return rand(B, T, H, 3 * D + 2)[..., 1:1 + 3 * D].split(D, dim=-1)
    return [rand(B, 1, H, D).expand(B, T, H, D) for _ in range(3)]  # "expanded": stride 0 over the tokens


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("kind", ["fused", "head_major", "misaligned", "expanded"])
@pytest.mark.parametrize("B,T,D", [(1, 1, 64), (2, 130, 64), (2, 129, 128)])
def test_strided_inputs_match_contiguous_ones(kind, B, T, D, dtype):
    H = 2
    views = _views(kind, B, T, H, D, dtype)
    results = []
    for prep in (lambda t: t.detach(), lambda t: t.detach().clone(memory_format=torch.contiguous_format)):
        q, k, v = [prep(t).requires_grad_() for t in views]
        out = m.sigmoid_attention(q, k, v, is_causal=True)
        results.append((out.detach(), *torch.autograd.grad(out.sum(), (q, k, v))))  # (an expanded output gradient)
    (o, dq, dk, dv), ref = results
    for a, b in zip((o, dk, dv), (ref[0], ref[2], ref[3])):  # computed in one order: bitwise
        assert torch.equal(a, b)
    assert torch.allclose(dq.float(), ref[1].float(), rtol=1e-2, atol=1e-4)  # order of the fp32 reductions


def test_inputs_changed_in_place_before_backward_are_refused():
    q, k, v = [torch.randn(1, 64, 2, 64, device="cuda", dtype=torch.bfloat16) for _ in range(3)]
    q.requires_grad_()
    out = m.sigmoid_attention(q, k, v)
    k.add_(1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.sum().backward()


def test_second_backward_needs_retain_graph():
    q = torch.randn(1, 64, 2, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    out = m.sigmoid_attention(q, q, q).sum()
    first, = torch.autograd.grad(out, q, retain_graph=True)
    second, = torch.autograd.grad(out, q)
    assert torch.equal(first, second)
    with pytest.raises(RuntimeError, match="backward through the graph a second time"):
        torch.autograd.grad(out, q)


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("dtype,dims", [(torch.bfloat16, (8, 24, 56, 72, 120)), (torch.float32, (4, 20, 60, 68, 124))])
def test_narrow_heads_match_zero_extended_ones(monkeypatch, dtype, dims, split):
    """Head dimensions below the kernels' 64 / 128 are read and written in place; padding them in memory gives the same."""
    if split:
        monkeypatch.setenv("SIGATTN_B200_BWD_SPLIT", "1")
    B, T, H = 2, 300, 3
    lens = torch.tensor([300, 131], dtype=torch.int32, device="cuda")
    for D in dims:
        g = torch.Generator(device="cuda").manual_seed(D)
        narrow = [torch.randn(B, T, H, D, device="cuda", generator=g).to(dtype) for _ in range(4)]
        wide = [torch.nn.functional.pad(t, (0, (64 if D <= 64 else 128) - D)) for t in narrow]
        res = []
        for q, k, v, do in (narrow, wide):
            q, k, v = [t.detach().requires_grad_() for t in (q, k, v)]
            out = m.sigmoid_attention_padded(q, k, v, seq_lens_k=lens, seq_lens_q=lens, is_causal=True, scale=0.3)
            res.append([t[..., :D] for t in (out.detach(), *torch.autograd.grad(out, (q, k, v), do))])
        for i, (a, b) in enumerate(zip(*res)):
            assert a.shape == narrow[0].shape
            # one order of operations except for dQ, whose fp32 reductions have none
            assert torch.equal(a, b) if i != 1 else torch.allclose(a.float(), b.float(), rtol=1e-2, atol=1e-4), (D, i)


@pytest.mark.parametrize("D", [64, 30])  # read in place, and through the Python path (zero-extended heads)
@pytest.mark.parametrize("requires_grad", [False, True])
@pytest.mark.parametrize("which", [0, 1, 2])
def test_forward_mode_is_refused(which, requires_grad, D):
    """A tangent cannot be propagated: an output without one would read as a derivative of zero."""
    args = [torch.randn(1, 64, 2, D, device="cuda", dtype=torch.bfloat16, requires_grad=requires_grad) for _ in range(3)]
    with torch.autograd.forward_ad.dual_level():
        args[which] = torch.autograd.forward_ad.make_dual(args[which], torch.ones_like(args[which]))
        with pytest.raises(NotImplementedError, match="forward-mode"):
            m.sigmoid_attention(*args)


def _varlen_call(q, k, v, mod):
    cu = torch.tensor([0, 70, 130], dtype=torch.int32, device="cuda")
    return m.sigmoid_attention_varlen(*(t.flatten(0, 1) for t in (q, k, v)), cu, cu, 70, 70, score_mod=mod.flatten())


def _padded_call(q, k, v, mod):
    lens = torch.tensor([65, 40], dtype=torch.int32, device="cuda")
    return m.sigmoid_attention_padded(q, k, v, seq_lens_k=lens, seq_lens_q=lens, is_causal=True, score_mod=mod)


_RELAYOUT = {
    # the same values, every eighth element of a row (the last stride is 8)
    "last_stride": lambda t: torch.stack([t] + [torch.full_like(t, 3)] * 7, -1)[..., 0],
    # rows two elements apart from 16-byte boundaries
    "misaligned": lambda t: torch.nn.functional.pad(t, (2, 0))[..., 2:],
    "contiguous": lambda t: t.contiguous(),
}


@pytest.mark.parametrize("call", [_padded_call, _varlen_call])
@pytest.mark.parametrize("how", sorted(_RELAYOUT))
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_saved_tensor_hooks_may_return_any_layout(how, call, dtype):
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = [torch.randn(2, 65, 2, 64, device="cuda", generator=g).to(dtype).requires_grad_() for _ in range(3)]
    mod = torch.randn(2, 65, device="cuda", generator=g)
    do = torch.randn(*call(q, k, v, mod).shape, device="cuda", generator=g).to(dtype)
    ref = torch.autograd.grad(call(q, k, v, mod), (q, k, v), do)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, _RELAYOUT[how]):
        out = call(q, k, v, mod)
    got = torch.autograd.grad(out, (q, k, v), do)
    for name, a, b in zip("qkv", got, ref):  # one key tile per (head, query tile): dQ has one order too
        assert torch.equal(a, b), name


def test_saved_tensor_hooks_that_change_what_was_saved_are_refused():
    """Another type, size or device than the forward had: an error, before a kernel gets a pointer."""
    q = torch.randn(2, 65, 2, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    mod = torch.zeros(2, 65, device="cuda")
    for unpack in (lambda t: t.half(), lambda t: t.cpu(), lambda t: t[..., :1]):
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: unpack(t) if t.dim() == 4 else t):
            out = m.sigmoid_attention(q, q, q, score_mod=mod)
        with pytest.raises(RuntimeError, match="sigmoid attention backward: query must be"):
            out.sum().backward()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t if t.dim() == 4 else t[:1]):
        out = m.sigmoid_attention(q, q, q, score_mod=mod)
    with pytest.raises(RuntimeError, match="score_mod must have 130 entries"):
        out.sum().backward()


def test_gradient_with_the_negative_bit():
    """A view whose values are the negated memory, with no strides to give it away."""
    q = torch.randn(2, 65, 2, 64, device="cuda", requires_grad=True)
    do = torch._neg_view(torch.randn(2, 65, 2, 64, device="cuda"))
    assert do.is_neg()
    got, = torch.autograd.grad(m.sigmoid_attention(q, q, q), q, do)
    ref, = torch.autograd.grad(m.sigmoid_attention(q, q, q), q, do.clone())
    assert torch.equal(got, ref)


def test_second_derivatives_are_refused():
    """create_graph is fine as long as nobody differentiates the gradients; then it is an error, not a missing term."""
    q, k, v = [torch.randn(2, 65, 2, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True) for _ in range(3)]
    plain = torch.autograd.grad(m.sigmoid_attention(q, k, v).float().square().sum(), (q, k, v))
    grads = torch.autograd.grad(m.sigmoid_attention(q, k, v).float().square().sum(), (q, k, v), create_graph=True)
    for a, b in zip(grads, plain):
        assert torch.equal(a, b)
    for g in grads:
        with pytest.raises(RuntimeError, match="differentiate sigmoid attention twice"):
            (g.float().sum() + q.float().sum()).backward(retain_graph=True)


@pytest.mark.parametrize("name", ["scale", "sigmoid_bias"])
def test_numbers_beyond_a_float_are_refused(name):
    q = torch.randn(1, 64, 2, 64, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(OverflowError):
        m.sigmoid_attention(q, q, q, **{name: 10 ** 400})


def test_an_output_without_a_gradient_gives_zeros():
    class NoGradient(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x):
            return x.sum()

        @staticmethod
        def backward(ctx, grad):
            return None

    qkv = [torch.randn(1, 64, 2, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True) for _ in range(3)]
    for g in torch.autograd.grad(NoGradient.apply(m.sigmoid_attention(*qkv)), qkv):
        assert g.shape == qkv[0].shape and g.abs().sum().item() == 0


@pytest.mark.parametrize("D", [64, 30])
@pytest.mark.parametrize("requires_grad", [False, True])
def test_tensor_subclasses_keep_their_type(D, requires_grad):
    class Tagged(torch.Tensor):
        pass

    q, k, v = [torch.randn(1, 64, 2, D, device="cuda", dtype=torch.bfloat16, requires_grad=requires_grad) for _ in range(3)]
    out = m.sigmoid_attention(q.as_subclass(Tagged), k, v)
    ref = m.sigmoid_attention(q, k, v)
    assert type(out) is Tagged and type(ref) is torch.Tensor
    assert type(m.sigmoid_attention(torch.nn.Parameter(q), k, v)) is torch.Tensor
    assert torch.equal(out.as_subclass(torch.Tensor), ref)
    if requires_grad:
        do = torch.randn_like(ref)
        for a, b in zip(torch.autograd.grad(out, (q, k, v), do), torch.autograd.grad(ref, (q, k, v), do)):
            assert torch.equal(a.as_subclass(torch.Tensor), b)


def test_switches_are_read_when_an_op_runs(monkeypatch):
    """Also by the backward, on autograd's thread, while another thread rewrites the environment."""
    import os
    import threading

    q, k, v, do = [torch.randn(2, 700, 2, 64, device="cuda", dtype=torch.bfloat16) for _ in range(4)]
    leaf = [t.requires_grad_() for t in (q, k, v)]
    monkeypatch.setenv("SIGATTN_B200_BWD_SPLIT", "1")
    split = torch.autograd.grad(m.sigmoid_attention(*leaf), leaf, do)
    monkeypatch.delenv("SIGATTN_B200_BWD_SPLIT")
    out = m.sigmoid_attention(*leaf)
    monkeypatch.setenv("SIGATTN_B200_BWD_SPLIT", "1")
    stop = threading.Event()

    def rewrite():
        i = 0
        while not stop.is_set():
            os.environ[f"SIGATTN_TEST_{i % 50}"] = "x" * (i % 7)
            i += 1

    other = threading.Thread(target=rewrite)
    other.start()
    try:
        for _ in range(20):
            for a, b in zip(torch.autograd.grad(out, leaf, do, retain_graph=True), split):
                assert torch.equal(a, b)  # the split backward is deterministic, dQ included
    finally:
        stop.set()
        other.join()
        for i in range(50):
            os.environ.pop(f"SIGATTN_TEST_{i}", None)
