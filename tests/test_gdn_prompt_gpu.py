"""Gated delta net kernels of prompts at the edges of their runs of rows, against the fp32 restatement."""
import numpy as np
import pytest
import torch

from sllm_b200.ops import gdn

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("taps", [2, 4, 8])
@pytest.mark.parametrize("counts", [[33], [40, 1, 0, 33, 2, 64], [5, 31, 32, 1, 1, 100], [0, 70, 0]])
@pytest.mark.parametrize("width", [514, 130])
def test_conv_rows(taps, counts, width):
    g = torch.Generator().manual_seed(taps + len(counts) + width)
    t, n = sum(counts), len(counts)
    off = torch.tensor([0] + list(np.cumsum(counts)), dtype=torch.int32)
    slots = torch.randperm(n + 2, generator=g)[:n].int()
    wide = torch.randn(t, width + 6, generator=g).bfloat16()
    w = (torch.randn(width, taps, generator=g) * 0.3).bfloat16()
    st = torch.randn(n + 2, taps - 1, width, generator=g).bfloat16()
    got_st = st.to(DEV)
    want = gdn.conv_silu(wide[:, 2:2 + width], w, st, off, slots)
    got = gdn.conv_silu(wide.to(DEV)[:, 2:2 + width], w.to(DEV), got_st, off.to(DEV), slots.to(DEV))
    assert (got.float().cpu() - want.float()).abs().max() <= 2.0 ** -7 * want.float().abs().max()      # one rounding of bf16
    assert torch.equal(got_st.cpu(), st)
