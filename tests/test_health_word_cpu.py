"""A kernel that finds the health word set leaves before its warps part.  They read the word at different times, and it may be
written meanwhile: unless they agree on one answer, some leave and the others wait for them - at a named barrier, which has no
limit, or with a tensor-memory address that the warp that left was to write."""

import os
import re

import pytest

from triton_sigmoid_b200._paths import CSRC

KERNELS = ["f32_tc_kernel.cuh", "fwd_kernel.cuh", "bwd_kernel.cuh", "bwd_stream_kernel.cuh"]


@pytest.mark.parametrize("name", KERNELS)
def test_early_return_is_one_answer_for_the_block(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    reads = re.findall(r".*&g_status_word\).*", text)
    assert reads
    for line in reads:
        kept = re.search(r"const bool (\w+) = ", line)
        assert "__syncthreads_or(" in line or (kept and re.search(r"__syncthreads_or\(%s\)" % kept.group(1), text)), line
