"""Rules that choose a kernel for prompts (host side)."""
from sllm_b200.ops import core


def test_prompt_tile_spreads_few_rows_and_fills_many():
    for scaled in (False, True):
        assert core._prompt_tile(130, 4096, scaled) == 64
        assert core._prompt_tile(8192, 28672, scaled) == 256
        for m in (129, 257, 1000, 5000):
            for n in (8, 1000, 4096):
                bn = core._prompt_tile(m, n, scaled)
                waves = lambda b: -(-(-(-m // 256) * -(-n // b)) // 74)
                assert all(waves(bn) * core._PROMPT_BLOCK[scaled][bn] <= waves(b) * core._PROMPT_BLOCK[scaled][b] for b in (64, 128, 256))
