"""Tensor-core prompt attention front end (kernel in csrc/prefill_attention.cu).

Sequences that start at position 0 and whose tokens are contiguous rows of the packed qkv activation, heads of 64, 128 or 256
channels, with or without a sliding window and sinks.  In a batch that also decodes, or continues prompts, the rows of the other
sequences read the paged cache.
"""
from __future__ import annotations

import math
from typing import Optional

import torch

from . import _lib
from .core import _alloc_q, _p, _stream, paged_attention, workspace

MIN_TOKENS = 128
TILE = 128


def _heads_fit(q, hd, qkv, sm_scale) -> bool:
    # (the kernel masks scores ahead of their scale, which must not turn them round)
    return ((sm_scale is None or sm_scale > 0) and q.is_cuda and qkv is not None and qkv.dtype == torch.bfloat16 and hd in (64, 128, 256) and not _lib.fake_active()
            and qkv.stride(1) == 1 and qkv.stride(0) == qkv.shape[1])


def usable(q, batch, hd, window, sinks, qkv, quant_out: bool = False, sm_scale: Optional[float] = None) -> bool:
    """Whether all rows of the batch take the kernel.  Results that are quantised to E4M3 are kept as they have been, since a last
    bit's difference moves them by a sixteenth: with a window or sinks they come from the pages."""
    if quant_out and (window or sinks is not None or hd != 128):
        return False
    return batch.cu_seqlens_host is not None and batch.max_seqlen >= MIN_TOKENS and _heads_fit(q, hd, qkv, sm_scale)


def fresh_part(q, batch, hd, qkv, sm_scale: Optional[float] = None) -> Optional[tuple]:
    """(sequences that take the kernel, [lo, hi) runs of the other rows) of a batch that mixes prompts with running requests, or
    None where no prompt of MIN_TOKENS starts in it."""
    if batch.row_off_host is None or batch.starts_host is None:
        return None
    if "fresh" not in batch.plans:
        off, fresh, rest = batch.row_off_host, [], []
        for i, start in enumerate(batch.starts_host):
            if off[i + 1] == off[i]:
                continue
            if start == 0 and off[i + 1] - off[i] >= MIN_TOKENS:
                fresh.append(i)
            elif rest and rest[-1][1] == off[i]:
                rest[-1][1] = off[i + 1]
            else:
                rest.append([off[i], off[i + 1]])
        batch.plans["fresh"] = (fresh, rest) if fresh else None
    part = batch.plans["fresh"]
    return part if part is not None and batch.row_off_host[-1] == q.shape[0] and _heads_fit(q, hd, qkv, sm_scale) else None


def build_tiles(cu_seqlens: list, device, rows: int = TILE, sequences: Optional[list] = None) -> torch.Tensor:
    """[num_tiles, 4] int32 = (first token row, sequence length, q0, 0); most work first."""
    tiles = []
    for s in sequences if sequences is not None else range(len(cu_seqlens) - 1):
        t0, n = cu_seqlens[s], cu_seqlens[s + 1] - cu_seqlens[s]
        for q0 in range(0, n, rows):
            tiles.append((t0, n, q0, 0))
    tiles.sort(key=lambda t: -t[2])
    return torch.tensor(tiles, dtype=torch.int32, device=device)


def prefill_attention(qkv, batch, hq, hkv, hd, *, sm_scale=None, quant_out=False, window=0, sinks=None, sequences=None):
    """Rows of the fresh ``sequences`` (default: all) -> [T, hq * hd], a QTensor with ``quant_out`` (heads of 128 without window and
    sinks); other rows of the result are not written."""
    t = qkv.shape[0]
    scale = sm_scale if sm_scale is not None else 1.0 / math.sqrt(hd)
    lib = _lib.kernels()
    rows = lib.sllm_prefill_tile_rows(hq, hkv, hd)
    key = ("prefill_tiles", rows, sequences is None)
    tiles = batch.plans.get(key)
    if tiles is None:
        cu = batch.cu_seqlens_host if sequences is None else batch.row_off_host
        tiles = batch.plans[key] = build_tiles(cu, qkv.device, rows, sequences)
    out = _alloc_q(t, hq * hd, qkv.device) if quant_out else torch.empty((t, hq * hd), dtype=torch.bfloat16, device=qkv.device)
    ob, o8, osc, ld = (None, out.data, out.scale, out.scale.stride(0)) if quant_out else (out, None, None, 0)
    if _lib.audit_enabled():
        _lib.record_dispatch("attention", "prefill_attention_kernel", rows=t, hq=hq, hkv=hkv, hd=hd, window=window,
                             grid=[hq // 2 if rows == TILE and hd != 256 else hq, tiles.shape[0]])
    rc = lib.sllm_prefill_attention(_p(qkv), t, qkv.stride(0), _p(tiles), tiles.shape[0], hq, hkv, hd, window, scale, _p(sinks),
                                    _p(ob), _p(o8), _p(osc), ld, _p(workspace(qkv.device).status), _stream())
    _lib.check(rc, "prefill_attention")
    return out


def mixed_attention(q, qkv, kv, batch, part, hq, hkv, hd, *, sm_scale=None, window=0, sinks=None):
    """Attention of a batch of which ``part`` (of ``fresh_part``) are fresh prompts; bf16 results."""
    fresh, rest = part
    out = prefill_attention(qkv, batch, hq, hkv, hd, sm_scale=sm_scale, window=window, sinks=sinks, sequences=fresh)
    if not rest:
        return out

    def paged(rows, seq_index, kv_lens, to=None):
        return paged_attention(rows, kv, batch.block_table, seq_index, kv_lens, hq, hkv, hd, window=window, sm_scale=sm_scale,
                               max_kv=batch.max_kv, sinks=sinks, out=to)

    if len(rest) == 1:
        lo, hi = rest[0]
        paged(q[lo:hi], batch.seq_index[lo:hi], batch.kv_lens[lo:hi], out[lo:hi])
        return out
    # rows in several runs: gathered, so that there is one launch however they lie
    if "paged_rows" not in batch.plans:
        idx = torch.tensor([r for lo, hi in rest for r in range(lo, hi)], device=q.device)
        batch.plans["paged_rows"] = (idx, batch.seq_index[idx], batch.kv_lens[idx])
    idx, seq_index, kv_lens = batch.plans["paged_rows"]
    out[idx] = paged(q[idx], seq_index, kv_lens)
    return out
