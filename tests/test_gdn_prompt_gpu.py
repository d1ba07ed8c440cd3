"""Gated delta net kernels of prompts at the edges of their runs of rows, against the fp32 restatement."""
import numpy as np
import pytest
import torch

from sllm_b200.ops import core, gdn

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


@pytest.mark.parametrize("ahead", [1, 31, 32, 70])
def test_conv_rows_ahead_of_the_first_sequence(ahead):
    """Offsets that do not start at row 0: the rows ahead belong to no sequence and no history is read for them."""
    counts, width, taps = [40, 33], 130, 4
    g = torch.Generator().manual_seed(ahead)
    t = ahead + sum(counts)
    off = torch.tensor([ahead] + [ahead + int(c) for c in np.cumsum(counts)], dtype=torch.int32)
    slots = torch.tensor([1, 0], dtype=torch.int32)
    x, w = torch.randn(t, width, generator=g).bfloat16(), (torch.randn(width, taps, generator=g) * 0.3).bfloat16()
    st = torch.randn(2, taps - 1, width, generator=g).bfloat16()
    got_st = st.to(DEV)
    want = gdn.conv_silu(x, w, st, off, slots)[ahead:].float()
    got = gdn.conv_silu(x.to(DEV), w.to(DEV), got_st, off.to(DEV), slots.to(DEV))[ahead:].float().cpu()
    assert (got - want).abs().max() <= 2.0 ** -7 * want.abs().max() and torch.equal(got_st.cpu(), st)


def test_recurrence_from_an_odd_element():
    """A contiguous qkv that starts between two 4-byte words: copied by the op, refused by the kernel's entry before any launch."""
    g = torch.Generator().manual_seed(3)
    t, qh, vh, hd = 40, 1, 2, 128
    rnd = lambda *s: torch.randn(*s, generator=g).bfloat16().to(DEV)
    qkv, z, b, a = rnd(t, (2 * qh + vh) * hd), rnd(t, vh * hd), rnd(t, vh), rnd(t, vh)
    a_log, dt, nw = rnd(vh).float(), rnd(vh), rnd(hd).float()
    off, slots = torch.tensor([0, t], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    flat = torch.zeros(qkv.numel() + 1, dtype=torch.bfloat16, device=DEV)
    flat[1:] = qkv.view(-1)
    odd = flat[1:].view(t, -1)
    assert odd.is_contiguous() and odd.data_ptr() % 4 == 2
    outs = []
    for x in (qkv, odd):
        st = torch.zeros(1, vh, hd, hd, device=DEV)
        outs.append((gdn.recurrent(x, z, b, a, a_log, dt, nw, st, off, slots, qh, vh), st))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    n = t * (2 * qh * hd + 2 * vh + vh * hd)
    scratch, out = torch.empty(n, device=DEV), torch.full((t, vh * hd), 7.0, dtype=torch.bfloat16, device=DEV)
    rc = gdn._k().sllm_gdn_recurrent_prompt(*(core._p(x) for x in (odd, z, b, a, a_log, dt, nw, outs[0][1], out, off, slots)), 1, t, qh, vh,
                                            hd, vh * hd, vh, core._p(scratch), n, core._stream())
    assert rc != 0 and (out == 7.0).all()
