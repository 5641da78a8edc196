"""The two tile shapes of the float32 kernels (chosen by how many 64-row tiles there are) at the edges of their tiles,
against the float64 oracle with the gates of tests/test_f32_gpu.py."""

import pytest
import torch

from tests.gpu_util import make_inputs
from tests.test_f32_gpu import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,T", [(1, 1, 15), (1, 2, 17), (1, 1, 81),          # 16-row tiles
                                   (1, 90, 63), (40, 2, 64), (1, 80, 65), (5, 9, 129)])  # 64-row tiles
def test_tile_edges(B, H, T, D, causal):
    q, k, v, do = make_inputs(B, T, T, H, D, torch.float32, std=0.5, seed=T + D, requires_grad=True)
    lens = torch.randint(1, T + 1, (B,), generator=torch.Generator().manual_seed(T), dtype=torch.int32)
    lens[0] = T
    with torch.no_grad():  # the oracle multiplies masked zeros with the padding: finite, but nothing a result may hold
        for t in (q, k, v, do):
            for b in range(B):
                t[b, int(lens[b]):] = 1.0e3
    lens = lens.cuda()
    _check(q, k, v, do, lens_q=lens, lens_k=lens, is_causal=causal, score_mod=torch.randn(B, T, device="cuda") * 0.5)
