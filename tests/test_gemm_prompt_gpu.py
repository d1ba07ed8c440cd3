"""The product of many rows (csrc/gemm_prompt.cu) at the edges of its tiles, against fp64."""
import pytest
import torch

from sllm_b200 import ops
from sllm_b200.ops import core
from sllm_b200.ops.core import LinearWeight

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _operands(m, n, k, scaled, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn(m, k, generator=g, device=DEV).bfloat16()
    w = (torch.randn(n, k, generator=g, device=DEV) * 0.05).bfloat16()
    r = torch.randn(m, n, generator=g, device=DEV).bfloat16()
    if not scaled:
        return x, LinearWeight("dense", w), x.double(), w.double(), r
    xq, wq = ops.quant_fp8(x), ops.quant_fp8(w)
    real = lambda q: q.data.view(torch.float8_e4m3fn).double() * q.scale.t().double().repeat_interleave(128, 1)[:, :k]
    return xq, LinearWeight("fp8", wq.data, wq.scale), real(xq), real(wq), r


def _close(got, want, xf, wf):
    # fp32 sums in any order (k 2^-23 of the sum of magnitudes) and one rounding to bf16
    bound = want.abs() * 2.0 ** -8 + (xf.abs() @ wf.abs().t()) * (xf.shape[1] * 2.0 ** -23) + 1e-30
    assert ((got.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("scaled", [False, True])
@pytest.mark.parametrize("m,n,k", [(129, 8, 64), (255, 264, 128), (257, 72, 208), (385, 520, 1040), (512, 256, 4096), (1030, 136, 640)])
@pytest.mark.parametrize("bn", [64, 128, 256])
def test_tiles(monkeypatch, scaled, m, n, k, bn):
    if bn not in core._PROMPT_BLOCK[scaled]:
        bn = 128                                        # bf16 has no tiles of 64 columns
    monkeypatch.setattr(core, "_prompt_tile", lambda *a: bn)
    x, w, xf, wf, r = _operands(m, n, k, scaled, m + n + k)
    want = xf @ wf.t()
    _close(ops.linear(x, w), want, xf, wf)
    _close(ops.linear(x, w, r), want + r.double(), xf, wf)
    assert ops.device_status(torch.device(DEV, 0)) == 0


@pytest.mark.parametrize("m,n,k", [(129, 8, 64), (300, 264, 128), (257, 520, 192), (385, 1032, 1040), (1030, 136, 4096), (2600, 8200, 320)])
@pytest.mark.parametrize("bn", [128, 256])
def test_partial_sums_are_those_of_the_general_product(monkeypatch, m, n, k, bn):
    """Two chains of K blocks, added in fp32: the same bits as the kernel that serves fewer rows."""
    monkeypatch.setattr(core, "_prompt_tile", lambda *a: bn)
    x, w, _, _, r = _operands(m, n, k, False, m + k)
    for res in (None, r):
        want = torch.empty(m, n, dtype=torch.bfloat16, device=DEV)
        core.gemm_raw(x, w.w, want, residual=res, transpose_out=False, bn=128, splits=1, stages=5)
        assert torch.equal(ops.linear(x, w, res), want)


def test_many_tiles_per_pair():
    """More tiles than pairs: accumulators, stages and scale chunks wrap around across tiles."""
    for scaled in (False, True):
        x, w, xf, wf, r = _operands(2600, 8200, 320, scaled, 5)
        _close(ops.linear(x, w, r), xf @ wf.t() + r.double(), xf, wf)


def test_activations_and_strided_rows():
    x, w, xf, wf, _ = _operands(300, 200, 256, False, 9)
    want = xf @ wf.t()
    relu = ops.linear(x, w, act="relu_sq").double()
    assert ((relu - want.clamp(min=0) ** 2).abs() <= (want.clamp(min=0) ** 2) * 2.0 ** -7 + 1e-3).all()
    cap = ops.linear(x, w, act="softcap", act_arg=2.0).double()
    assert ((cap - 2.0 * torch.tanh(want / 2.0)).abs() <= 2.0 ** -7).all()
    wide = torch.zeros(300, 512, device=DEV, dtype=torch.bfloat16)
    wide[:, 8:264] = x
    _close(ops.linear(wide[:, 8:264], w), want, xf, wf)


@pytest.mark.parametrize("m", [1, 128, 129, 300])
@pytest.mark.parametrize("cap", [0.0, -1.0, float("nan")])
def test_a_soft_cap_that_is_not_positive_is_refused(m, cap):
    x, w, _, _, _ = _operands(m, 64, 64, False, 1)
    with pytest.raises(ops.KernelError):
        ops.linear(x, w, act="softcap", act_arg=cap)


@pytest.mark.parametrize("m", [128, 129, 300])
@pytest.mark.parametrize("k", [64, 128])
def test_scales_of_one_block_with_any_leading_stride(m, k):
    """One K block: the transposed scales of a file are [1, n] with a leading stride of 1."""
    x, w, xf, wf, _ = _operands(m, 72, k, True, k)
    turned = lambda s: torch.empty(s.shape[1], 1, device=DEV).copy_(s.t()).t().contiguous()
    xt, wt = ops.QTensor(x.data, turned(x.scale)), LinearWeight("fp8", w.w, turned(w.scale_t))
    assert xt.scale.stride(0) == 1 and wt.scale_t.stride(0) == 1
    _close(ops.linear(xt, wt), xf @ wf.t(), xf, wf)
