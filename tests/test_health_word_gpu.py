"""Kernels that are launched while the health word is set (here: from a captured graph, which the host does not look at) return
at once and leave their outputs alone; once the word has been read and cleared they compute."""

import pytest
import torch

import triton_sigmoid_b200 as m
from tests.gpu_util import launch_form, make_inputs
from triton_sigmoid_b200 import _cabi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split_backward", [False, True])
@pytest.mark.parametrize("B,T,H,D,dtype,form", [
    (1, 512, 2, 64, torch.float32, _cabi.FORM_F32_TC),
    (1, 512, 16, 128, torch.float32, _cabi.FORM_F32_TC),
    (1, 512, 2, 64, torch.float16, _cabi.FORM_BWD),           # forward: keys split over a cluster
    (16, 256, 16, 128, torch.bfloat16, _cabi.FORM_BWD),       # persistent forward
    (80, 256, 16, 64, torch.bfloat16, _cabi.FORM_BWD_BY_HEAD),
])
def test_replay_while_the_word_is_set(B, T, H, D, dtype, form, split_backward, monkeypatch):
    lib = _cabi.load()
    assert launch_form(B, H, T, T, D, dtype, True) == form
    assert m.device_status() == 0
    if split_backward:
        if dtype == torch.float32:
            pytest.skip("an option of the 16-bit kernels")
        monkeypatch.setenv("SIGATTN_B200_BWD_SPLIT", "1")
        form = None
    q, k, v, do = make_inputs(B, T, T, H, D, dtype, std=0.5, seed=1, requires_grad=True)

    def step():
        out = m.sigmoid_attention(q, k, v)
        return (out,) + torch.autograd.grad(out, (q, k, v), do)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        want = [t.detach().clone() for t in step()]
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = [t.detach() for t in step()]
    looked_at = [0, 2, 3] if form == _cabi.FORM_BWD else [0, 1, 2, 3]  # (dQ comes from another kernel in this form)
    for t in got:
        t.fill_(7.0)
    torch.cuda.synchronize()
    assert lib.sigattn_selftest_bounded_wait(0, 10) == 1, lib.sigattn_last_error()
    graph.replay()
    torch.cuda.synchronize()
    assert all((got[i] == 7.0).all() for i in looked_at)
    assert m.device_status() == 0x30001
    graph.replay()
    torch.cuda.synchronize()
    assert m.device_status() == 0
    for i in looked_at:
        assert ((got[i].double() - want[i].double()).norm() / want[i].double().norm()).item() <= (1e-5 if dtype == torch.float32 else 1e-2)
