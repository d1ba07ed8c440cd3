"""Rules that choose a kernel for prompts (host side)."""
import pytest
import torch

from sllm_b200.ops import core, moe, w4
from sllm_b200.ops.w4 import W4Weight
from sllm_b200.parallel.ep import NcclEP, NoEP


def test_prompt_tile_spreads_few_rows_and_fills_many():
    for scaled in (False, True):
        assert core._prompt_tile(130, 4096, scaled) == (64 if scaled else 128)       # bf16: 64 columns are no faster than 128
        assert core._prompt_tile(8192, 28672, scaled) == 256
        for m in (129, 257, 1000, 5000):
            for n in (8, 1000, 4096):
                bn = core._prompt_tile(m, n, scaled)
                waves = lambda b: -(-(-(-m // 256) * -(-n // b)) // 74)
                assert all(waves(bn) * core._PROMPT_BLOCK[scaled][bn] <= waves(b) * core._PROMPT_BLOCK[scaled][b] for b in core._PROMPT_BLOCK[scaled])


def test_group_tile_holds_the_mean_of_the_groups():
    assert [w4._group_tile(rows, 4096, 128) for rows in (64, 3000, 3400, 7936, 9900, 9950)] == [16, 32, 64, 96, 96, 128]
    assert w4._group_tile(64, 16, 128) == 16                      # no group has more rows than the call has tokens
    assert w4._group_tile(7936, 80, 128) == 96


@pytest.mark.parametrize("ranks", [1, 2, 8])
def test_group_tile_of_a_rank_is_that_of_the_whole_layer(monkeypatch, ranks):
    """The rows that a rank permutes are those of all experts, its weight holds only its own."""
    experts, k, t, d = 16, 4, 24, 128
    g = torch.Generator().manual_seed(1)
    seen = []

    def product(x, w, tok_off=None, max_group_tokens=None, tok_scale=None, row_ptr=None, experts=0):
        seen.append(w4._group_tile(40 * x.shape[0], 40 * max_group_tokens, experts or w.groups))
        return torch.zeros(x.shape[0], w.n)

    monkeypatch.setattr(moe, "linear_w4", product)
    ep = NoEP() if ranks == 1 else NcclEP(ranks, 1, "cpu")
    ep.combine = lambda yp, dst, residual: yp
    lo, hi = ep.expert_range(experts)
    local = hi - lo
    gate_up, down = (W4Weight.quantize("mxfp4", torch.randn(local, n, kk, generator=g)) for n, kk in ((2 * d, d), (d, d)))
    idx = torch.stack([torch.randperm(experts, generator=g)[:k] for _ in range(t)]).int()
    ep.experts_combine(torch.randn(t, d, generator=g), idx, torch.full((t, k), 0.25), gate_up, down, "silu", lo, hi, None)
    assert seen == [w4._group_tile(40 * t * k, 40 * t, experts)] * 2
