"""Prompt attention (csrc/prefill_attention.cu) over head widths, groups, windows, sinks and ragged lengths, against fp64."""
import math

import pytest
import torch

from sllm_b200 import ops
from sllm_b200.engine.batch import make_prefill_batch
from sllm_b200.ops import _lib, prefill
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


def _close(got, want, roundings=1):
    """One rounding to bf16 (or two, against a result that is rounded itself) is all that separates a result from 64 bits: at most
    2^-8 of a value, and in the norm what the rounded exact values show; probabilities with 8 bits add 6 % and more to it."""
    got = got.double()
    assert (got - want).abs().max() <= roundings * (2.0 ** -8 + 2.0 ** -13) * want.abs().max()
    if roundings == 1:
        assert (got - want).norm() <= 1.01 * (want.bfloat16().double() - want).norm()
    else:
        assert (got - want).norm() / want.norm() < 2.0 ** -8


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
    if hd == 128 and not window and sinks is None:
        q = prefill.prefill_attention(qkv, b, hq, hkv, hd, quant_out=True)
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
    _close(ops.attention(q, kv, b, hq, hkv, hd, qkv=qkv), want, 2)


@pytest.mark.parametrize("hd", [64, 128, 256])
def test_subnormal_probabilities_stay(hd):
    """Every other key's probability is 2^-130 of the largest; its values are so large that they are all of the result."""
    n, hq, hkv = 300, 4, 2
    qkv = torch.zeros(n, hq + 2 * hkv, hd, device=DEV)
    qkv[:, :hq, 0] = 1.0
    qkv[1::2, hq:hq + hkv, 0] = -130.0
    qkv[1::2, hq + hkv:] = 2.0 ** 120
    qkv = qkv.view(n, -1).bfloat16()
    b = make_prefill_batch([[0] * n], torch.zeros((1, 1), dtype=torch.int32, device=DEV), DEV)
    got = prefill.prefill_attention(qkv, b, hq, hkv, hd, sm_scale=math.log(2.0)).double()
    row = torch.arange(n, device=DEV, dtype=torch.double)[:, None]
    want = ((row + 1) / 2).floor() / (row / 2 + 1).floor() * 2.0 ** -10
    # a subnormal of 2^-130 has 19 bits, its exponent an error of 130 2^-23; then one rounding
    assert ((got - want).abs() <= want * (2.0 ** -8 + 2.0 ** -14)).all()


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("hq,hkv", [(2, 2), (4, 1)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("window", [0, 100])
def test_a_request_does_not_reach_its_neighbours(hd, hq, hkv, value, window):
    """Rows of a request whose values are not finite lie behind another request's in the last tile of keys."""
    lens = [129, 140, 257, 1, 383]
    g = torch.Generator(device=DEV).manual_seed(hd + hq)
    qkv = torch.randn(sum(lens), (hq + 2 * hkv) * hd, generator=g, device=DEV).bfloat16()
    b = make_prefill_batch([[0] * n for n in lens], torch.zeros((len(lens), 1), dtype=torch.int32, device=DEV), DEV)
    broken = qkv.clone()
    broken[129:129 + 140, hq * hd:] = value                # keys and values of the second and the fourth
    broken[129 + 140 + 257, hq * hd:] = value
    keep = torch.cat([torch.full((n,), i not in (1, 3), device=DEV) for i, n in enumerate(lens)])
    for quant in (False, True) if hd == 128 and not window else (False,):
        want, got = (prefill.prefill_attention(x, b, hq, hkv, hd, window=window, quant_out=quant) for x in (qkv, broken))
        if quant:
            assert torch.equal(got.data[keep], want.data[keep]) and torch.equal(got.scale[:, keep], want.scale[:, keep])
        else:
            assert want.isfinite().all() and torch.equal(got[keep], want[keep])


def test_a_request_does_not_reach_its_neighbours_in_a_mixed_batch():
    hq, hkv, hd, page = 8, 2, 128, 16
    starts, counts = [0, 77, 0, 40, 0], [300, 1, 140, 33, 150]
    g = torch.Generator(device=DEV).manual_seed(4)
    t, blocks = sum(counts), 320 // page
    qkv = torch.randn(t, (hq + 2 * hkv) * hd, generator=g, device=DEV).bfloat16()
    results = []
    for bad in (False, True):
        kv = KVLayer(*(torch.ones(5 * blocks, hkv, page, hd, device=DEV).bfloat16() for _ in range(2)), None, None, False, page)
        table = torch.arange(5 * blocks, dtype=torch.int32, device=DEV).view(5, blocks)
        b = make_prefill_batch([[0] * c for c in counts], table, DEV, starts)
        x = qkv.clone()
        if bad:
            x[300, (hq + hkv) * hd:] = float("inf")          # the second request's only row
            x[441:474, (hq + hkv) * hd:] = float("nan")      # the fourth's
        q = ops.rope_kv_append(x, b.positions, b.seq_index, b.block_table, kv, hq, hkv, hd, 1e4)
        assert prefill.fresh_part(q, b, hd, x)[0] == [0, 2, 4]
        results.append(ops.attention(q, kv, b, hq, hkv, hd, qkv=x))
    keep = torch.cat([torch.full((c,), i not in (1, 3), device=DEV) for i, c in enumerate(counts)])
    assert torch.equal(results[0][keep], results[1][keep])


def test_rows_between_prompts_take_one_launch():
    """Prompts and other rows in turn: the others are gathered for the pages."""
    hq, hkv, hd, page = 8, 2, 128, 16
    starts, counts = [5, 0, 77, 0, 40, 0, 3, 0, 9], [1, 300, 1, 129, 20, 150, 2, 128, 1]
    g = torch.Generator(device=DEV).manual_seed(6)
    t, blocks = sum(counts), 320 // page
    kv = KVLayer(*(torch.randn(9 * blocks, hkv, page, hd, generator=g, device=DEV).bfloat16() for _ in range(2)), None, None, False, page)
    table = torch.arange(9 * blocks, dtype=torch.int32, device=DEV).view(9, blocks)
    b = make_prefill_batch([[0] * c for c in counts], table, DEV, starts)
    qkv = torch.randn(t, (hq + 2 * hkv) * hd, generator=g, device=DEV).bfloat16()
    q = ops.rope_kv_append(qkv, b.positions, b.seq_index, b.block_table, kv, hq, hkv, hd, 1e4)
    want = ops.paged_attention(q, kv, table, b.seq_index, b.kv_lens, hq, hkv, hd, max_kv=b.max_kv).double()
    for _ in range(2):                                  # the second call (another layer) uses the same plans
        _lib.dispatch_records(clear=True)
        _lib.audit(True)
        try:
            got = ops.attention(q, kv, b, hq, hkv, hd, qkv=qkv)
        finally:
            _lib.audit(False)
        assert [e["kernel"] for e in _lib.dispatch_records(clear=True)] == ["prefill_attention_kernel", "paged_attention_kernel"]
        _close(got, want, 2)


@pytest.mark.parametrize("scale", [0.0, -0.2, 0.2])
@pytest.mark.parametrize("hd,window", [(64, 0), (128, 0), (128, 50), (256, 0)])
def test_any_scale(scale, hd, window):
    """Scores may be turned round or levelled by their scale."""
    hq, hkv, page, lens = 4, 2, 16, [200, 33]
    g = torch.Generator(device=DEV).manual_seed(hd)
    kv = KVLayer(*(torch.zeros(26, hkv, page, hd, device=DEV).bfloat16() for _ in range(2)), None, None, False, page)
    b = make_prefill_batch([[0] * n for n in lens], torch.arange(26, dtype=torch.int32, device=DEV).view(2, 13), DEV)
    qkv = torch.randn(sum(lens), (hq + 2 * hkv) * hd, generator=g, device=DEV).bfloat16()
    q = ops.rope_kv_append(qkv, b.positions, b.seq_index, b.block_table, kv, hq, hkv, hd, 1e4)
    got = ops.attention(q, kv, b, hq, hkv, hd, qkv=qkv, window=window, sm_scale=scale)
    turned = qkv.double()
    turned[:, :hq * hd] *= scale * math.sqrt(hd)
    _close(got, _want(turned, lens, hq, hkv, hd, window, None))


@pytest.mark.parametrize("hd", [64, 256])
def test_quantised_results_of_other_heads_are_refused(hd):
    """As by the pages, which need heads of 128 for them."""
    hq, hkv, n = 4, 2, 200
    kv = KVLayer(*(torch.zeros(13, hkv, 16, hd, device=DEV).bfloat16() for _ in range(2)), None, None, False, 16)
    b = make_prefill_batch([[0] * n], torch.arange(13, dtype=torch.int32, device=DEV).view(1, 13), DEV)
    qkv = torch.zeros(n, (hq + 2 * hkv) * hd, dtype=torch.bfloat16, device=DEV)
    with pytest.raises(ValueError):
        ops.attention(qkv[:, :hq * hd], kv, b, hq, hkv, hd, qkv=qkv, quant_out=True)
