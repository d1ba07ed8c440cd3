"""Rotation and page append, a warp per head (csrc/elementwise.cu), against the fp32 restatement: both grids, every head width."""
import pytest
import torch

from sllm_b200 import ops
from sllm_b200.ops.core import KVLayer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [1, 37, 600])
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("hq,hkv,hd,rd", [(3, 1, 64, 64), (8, 2, 128, 128), (4, 4, 256, 64), (2, 1, 96, 30), (2, 2, 320, 320), (9, 3, 34, 34)])
def test_rows(tokens, fp8, hq, hkv, hd, rd):
    g = torch.Generator().manual_seed(tokens + hd)
    qkv = torch.randn(tokens, (hq + 2 * hkv) * hd, generator=g).bfloat16()
    qkv[0, hq * hd:(hq + hkv) * hd] = 0                     # an all-zero key: scale 1
    pos = torch.arange(tokens, dtype=torch.int32) * 3
    pages = tokens * 3 // 16 + 1
    seq = torch.zeros(tokens, dtype=torch.int32)
    table = torch.randperm(pages, generator=g).int()[None]

    def layer(dev):
        v = lambda: torch.zeros(pages, hkv, 16, hd, dtype=torch.uint8 if fp8 else torch.bfloat16, device=dev)
        s = lambda: torch.zeros(pages, hkv, 16, device=dev) if fp8 else None
        return KVLayer(v(), v(), s(), s(), fp8, 16)
    want_kv, kv = layer("cpu"), layer("cuda")
    want = ops.rope_kv_append(qkv.clone(), pos, seq, table, want_kv, hq, hkv, hd, 10000.0, rd)
    mine = qkv.cuda()
    got = ops.rope_kv_append(mine, pos.cuda(), seq.cuda(), table.cuda(), kv, hq, hkv, hd, 10000.0, rd)
    # angles of up to 1800 radians in fp32 are off by 1e-4; a rounding to bf16 by 2^-8 of the value
    close = lambda a, b: (a.float().cpu() - b.float()).abs().max() <= 2.0 ** -8 * b.float().abs().max() + 2e-3
    assert close(got, want)
    if fp8:
        for a, b, sa, sb in ((kv.k, want_kv.k, kv.k_scale, want_kv.k_scale), (kv.v, want_kv.v, kv.v_scale, want_kv.v_scale)):
            x = a.cpu().view(torch.float8_e4m3fn).float() * sa.cpu()[..., None]
            y = b.view(torch.float8_e4m3fn).float() * sb[..., None]
            assert ((x - y).abs() <= y.abs() * 2.0 ** -3 + sb[..., None] * 2.0 ** -8 + 2e-3).all()       # one E4M3 step
            assert torch.allclose(sa.cpu(), sb, rtol=2.0 ** -6)
    else:
        assert close(kv.k, want_kv.k) and torch.equal(kv.v.cpu(), want_kv.v)
