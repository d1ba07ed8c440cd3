"""Prompt attention (csrc/prefill_attention.cu) over head widths, groups, windows, sinks and ragged lengths, against fp64."""
import math

import pytest
import torch

from sllm_b200 import ops
from sllm_b200.engine.batch import make_prefill_batch
from sllm_b200.ops import prefill
from sllm_b200.ops.core import KVLayer

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _want(qkv, lens, hq, hkv, hd, window, sinks):
    x = qkv.double().view(-1, hq + 2 * hkv, hd)
    out, t0 = [], 0
    for n in lens:
        q, k, v = x[t0:t0 + n, :hq], x[t0:t0 + n, hq:hq + hkv], x[t0:t0 + n, hq + hkv:]
        k, v = (y.repeat_interleave(hq // hkv, 1) for y in (k, v))
        s = torch.einsum("qhd,khd->hqk", q, k) / math.sqrt(hd)
        gap = torch.arange(n, device=DEV)[:, None] - torch.arange(n, device=DEV)[None]
        s = s.masked_fill((gap < 0) | ((gap >= window) if window else False), float("-inf"))
        if sinks is not None:
            s = torch.cat([s, sinks.double()[:, None, None].expand(hq, n, 1)], -1)
        out.append(torch.einsum("hqk,khd->qhd", torch.softmax(s, -1)[..., :n], v).reshape(n, hq * hd))
        t0 += n
    return torch.cat(out)


def _close(got, want):
    # probabilities and results are rounded to bf16: 2^-9 of their size each, sums of many rounding errors below that
    got = got.double()
    assert (got - want).norm() / want.norm() < 2.0 ** -7
    assert (got - want).abs().max() <= 2.0 ** -6 * want.abs().max()


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("hq,hkv", [(4, 4), (3, 1), (4, 2), (8, 1)])
@pytest.mark.parametrize("window,with_sinks", [(0, False), (0, True), (100, True), (128, False), (1, False)])
@pytest.mark.parametrize("lens", [[128], [1, 129, 257, 64], [700, 383]])
def test_forms(hd, hq, hkv, window, with_sinks, lens):
    g = torch.Generator(device=DEV).manual_seed(hd + hq + window + len(lens))
    qkv = torch.randn(sum(lens), (hq + 2 * hkv) * hd, generator=g, device=DEV)
    qkv[:, :hq * hd] *= 3.0                             # maxima that grow by more than the rescaling threshold along a row
    qkv = qkv.bfloat16()
    sinks = torch.randn(hq, generator=g, device=DEV) * 2 if with_sinks else None
    b = make_prefill_batch([[0] * n for n in lens], torch.zeros((len(lens), 1), dtype=torch.int32, device=DEV), DEV)
    assert prefill.usable(qkv, b, hd, window, sinks, qkv)
    want = _want(qkv, lens, hq, hkv, hd, window, sinks)
    _close(prefill.prefill_attention(qkv, b, hq, hkv, hd, window=window, sinks=sinks), want)
    if hd == 128:
        q = prefill.prefill_attention(qkv, b, hq, hkv, hd, window=window, sinks=sinks, quant_out=True)
        got = q.data.view(torch.float8_e4m3fn).double() * q.scale.t().double().repeat_interleave(128, 1)
        assert (got - want).norm() / want.norm() < 2.0 ** -4
    assert ops.device_status(torch.device(DEV, 0)) == 0


def test_scores_that_keep_growing():
    """Every tile's maximum lies far above the last one's: O is rescaled in each."""
    n, hq, hkv, hd = 640, 2, 1, 128
    g = torch.Generator(device=DEV).manual_seed(1)
    qkv = torch.randn(n, (hq + 2 * hkv) * hd, generator=g, device=DEV)
    qkv[:, :hq * hd] = 1.0
    qkv[:, hq * hd:(hq + 1) * hd] = torch.linspace(0, 20, n, device=DEV)[:, None]
    qkv = qkv.bfloat16()
    b = make_prefill_batch([[0] * n], torch.zeros((1, 1), dtype=torch.int32, device=DEV), DEV)
    _close(prefill.prefill_attention(qkv, b, hq, hkv, hd), _want(qkv, [n], hq, hkv, hd, 0, None))


def test_prompts_beside_running_requests():
    """Fresh prompts of a mixed batch take the kernel, short ones, continued ones and single tokens read the pages."""
    hq, hkv, hd, page = 8, 2, 128, 16
    starts, counts = [0, 77, 0, 40, 0], [300, 1, 20, 33, 150]
    g = torch.Generator(device=DEV).manual_seed(3)
    t, total = sum(counts), max(s + c for s, c in zip(starts, counts))
    blocks = total // page + 1
    kv = KVLayer(*(torch.randn(5 * blocks, hkv, page, hd, generator=g, device=DEV).bfloat16() for _ in range(2)), None, None, False, page)
    table = torch.arange(5 * blocks, dtype=torch.int32, device=DEV).view(5, blocks)
    b = make_prefill_batch([[0] * c for c in counts], table, DEV, starts)
    qkv = torch.randn(t, (hq + 2 * hkv) * hd, generator=g, device=DEV).bfloat16()
    q = ops.rope_kv_append(qkv, b.positions, b.seq_index, b.block_table, kv, hq, hkv, hd, 1e4)
    part = prefill.fresh_part(q, b, hd, qkv)
    assert part == ([0, 4], [[300, 354]])
    want = ops.paged_attention(q, kv, table, b.seq_index, b.kv_lens, hq, hkv, hd, max_kv=b.max_kv).double()
    _close(ops.attention(q, kv, b, hq, hkv, hd, qkv=qkv), want)
