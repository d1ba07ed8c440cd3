"""4-bit weights with many rows: expanded dense matrices and the token tiles of routed experts."""
import numpy as np
import pytest
import torch

from sllm_b200 import ops
from sllm_b200.ops import _lib, w4
from sllm_b200.ops.w4 import W4Weight, linear_w4

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("fmt", ["mxfp4", "nvfp4"])
@pytest.mark.parametrize("t,n,k", [(129, 136, 200), (260, 640, 384), (300, 1032, 128)])
def test_expanded_products(monkeypatch, fmt, t, n, k):
    g = torch.Generator(device=DEV).manual_seed(t)
    weight = W4Weight.quantize_device(fmt, torch.randn(n, k, generator=g, device=DEV) * 0.05)
    real = weight.dequantized(0).double().to(DEV)
    x = torch.randn(t, k, generator=g, device=DEV).bfloat16()
    r = torch.randn(t, n, generator=g, device=DEV).bfloat16()
    for elements in (w4.EXPAND_ELEMENTS, 256 * k):                 # at once, and in pieces of 256 rows
        monkeypatch.setattr(w4, "EXPAND_ELEMENTS", elements)
        for res in (None, r):
            want = x.double() @ real.t() + (0 if res is None else res.double())
            bound = want.abs() * 2.0 ** -8 + (x.double().abs() @ real.abs().t()) * (k * 2.0 ** -23)
            assert ((linear_w4(x, weight, residual=res).double() - want).abs() <= bound).all()
    assert ops.device_status(torch.device(DEV, 0)) == 0


@pytest.mark.parametrize("fmt", ["mxfp4", "nvfp4"])
@pytest.mark.parametrize("t,n,k", [(129, 136, 64), (260, 640, 200), (300, 1032, 384), (1076, 4096, 4096)])
def test_expanded_products_have_the_bits_of_packed_ones(fmt, t, n, k):
    """Four chains of K blocks, added in fp32, on both sides."""
    g = torch.Generator(device=DEV).manual_seed(t)
    weight = W4Weight.quantize_device(fmt, torch.randn(n, k, generator=g, device=DEV) * 0.05)
    x = torch.randn(t, k, generator=g, device=DEV).bfloat16()
    r = torch.randn(t, n, generator=g, device=DEV).bfloat16()
    for res in (None, r):
        assert torch.equal(linear_w4(x, weight, residual=res), linear_w4(x, weight, residual=res, splits=1))


def test_no_room_for_expanded_weights(monkeypatch):
    """A product whose weight cannot be expanded for want of memory takes the packed kernel."""
    g = torch.Generator(device=DEV).manual_seed(2)
    weight = W4Weight.quantize_device("nvfp4", torch.randn(19200, 256, generator=g, device=DEV) * 0.05)
    x = torch.randn(300, 256, generator=g, device=DEV).bfloat16()
    want = linear_w4(x, weight)

    def full(*a, **k):
        raise torch.OutOfMemoryError("no room")

    with monkeypatch.context() as m:
        m.setattr(w4.torch, "empty", lambda *a, **k: full() if a[0] == (19200, 256) else torch.zeros(*a, **k))
        _lib.dispatch_records(clear=True)
        _lib.audit(True)
        try:
            got = linear_w4(x, weight)
        finally:
            _lib.audit(False)
    assert [e["kernel"] for e in _lib.dispatch_records(clear=True)] == ["gemm_w4_kernel"]
    assert torch.equal(got, want)


@pytest.mark.parametrize("counts", [[0, 0, 300], [17, 0, 64, 65, 1, 128, 0, 129], [3] * 70, [0] * 40 + [200, 5]])
def test_token_tiles_of_experts(counts):
    g = torch.Generator(device=DEV).manual_seed(len(counts))
    e, t, n, k = len(counts), sum(counts), 136, 256
    weight = W4Weight.quantize_device("mxfp4", torch.randn(e, n, k, generator=g, device=DEV) * 0.05)
    off = torch.tensor([0] + list(np.cumsum(counts)), dtype=torch.int32, device=DEV)
    x = torch.randn(t, k, generator=g, device=DEV).bfloat16()
    scale = torch.rand(t, generator=g, device=DEV)
    want, size = torch.zeros(t, n, dtype=torch.double, device=DEV), torch.zeros(t, n, dtype=torch.double, device=DEV)
    for i in range(e):
        a, b = int(off[i]), int(off[i + 1])
        if b > a:
            real = weight.dequantized(i).double().to(DEV)
            want[a:b] = x[a:b].double() @ real.t() * scale[a:b, None].double()
            size[a:b] = x[a:b].double().abs() @ real.abs().t() * scale[a:b, None].double()
    for splits in (0, 1, 2):
        got = linear_w4(x, weight, tok_off=off, tok_scale=scale, max_group_tokens=t, splits=splits).double()
        assert ((got - want).abs() <= want.abs() * 2.0 ** -8 + size * (k * 2.0 ** -23)).all()
    assert ops.device_status(torch.device(DEV, 0)) == 0


def _audited(call):
    _lib.dispatch_records(clear=True)
    _lib.audit(True)
    try:
        y = call()
    finally:
        _lib.audit(False)
    return y, _lib.dispatch_records(clear=True)


@pytest.mark.parametrize("fmt", ["mxfp4", "nvfp4"])
@pytest.mark.parametrize("t", [65, 95, 96])
@pytest.mark.parametrize("n,k,splits", [(136, 200, 0), (264, 1024, 1), (264, 1024, 4)])
def test_dense_tile_of_96_columns(fmt, t, n, k, splits):
    g = torch.Generator(device=DEV).manual_seed(t + n)
    weight = W4Weight.quantize_device(fmt, torch.randn(n, k, generator=g, device=DEV) * 0.05)
    real = weight.dequantized(0).double().to(DEV)
    x = torch.randn(t, k, generator=g, device=DEV).bfloat16()
    r = torch.randn(t, n, generator=g, device=DEV).bfloat16()
    for res in (None, r):
        got, records = _audited(lambda: linear_w4(x, weight, residual=res, splits=splits))
        assert [(e["kernel"], e["bn"]) for e in records] == [("gemm_w4_kernel", 96)]
        want = x.double() @ real.t() + (0 if res is None else res.double())
        bound = want.abs() * 2.0 ** -8 + (x.double().abs() @ real.abs().t()) * (k * 2.0 ** -23)
        assert ((got.double() - want).abs() <= bound).all()
    assert ops.device_status(torch.device(DEV, 0)) == 0


@pytest.mark.parametrize("fmt", ["mxfp4", "nvfp4"])
@pytest.mark.parametrize("counts", [[0, 95, 96, 97, 193, 1, 0, 40] * 5 + [0] * 30 + [65] * 10, [96, 0, 97, 30], [0] * 33 + [193, 0, 95]])
@pytest.mark.parametrize("splits", [0, 1, 2])
def test_grouped_tile_of_96_columns(fmt, counts, splits):
    """Groups below, at and above one and two tiles, in lists that the tile lookup walks 32 groups at a time."""
    e, t, n, k = len(counts), sum(counts), 136, 256
    g = torch.Generator(device=DEV).manual_seed(e)
    weight = W4Weight.quantize_device(fmt, torch.randn(e, n, k, generator=g, device=DEV) * 0.05)
    off = torch.tensor([0] + list(np.cumsum(counts)), dtype=torch.int32, device=DEV)
    x = torch.randn(t, k, generator=g, device=DEV).bfloat16()
    experts = 5 * t // (4 * 80)                          # such that the mean with a quarter to spare is about 80
    got, records = _audited(lambda: linear_w4(x, weight, tok_off=off, max_group_tokens=t, splits=splits, experts=experts))
    assert [(r["kernel"], r["bn"]) for r in records] == [("gemm_w4_kernel", 96)]
    for i in range(e):
        a, b = int(off[i]), int(off[i + 1])
        if b > a:
            real = weight.dequantized(i).double().to(DEV)
            want, size = x[a:b].double() @ real.t(), x[a:b].double().abs() @ real.abs().t()
            assert ((got[a:b].double() - want).abs() <= want.abs() * 2.0 ** -8 + size * (k * 2.0 ** -23)).all(), i
    assert ops.device_status(torch.device(DEV, 0)) == 0
