"""Attention of the true 32-bit path over one step's batch (csrc/attention_f32.cu): prompt portions by tiles of 64 query
rows, single tokens by spans of the context.  Both sum a query in the same order: a token's result is the same bits
whichever kernel takes it."""
from __future__ import annotations

from ctypes import c_float, c_int

import torch

from . import attention_mma
from .ops import KernelError, _check, _need, _p, _stream, check_pages, core

SPAN = 256                       # keys a span, the same number as in the source
HEAD_DIMS = (32, 64, 128)
MOST_GROUP = 64                  # query heads per kv head of the tile kernel: its rows
MOST_SINGLE_GROUP = 8            # ... of the span kernel
#: Bytes of partial sums the span kernel's buffer may have.  They are sized by the longest context times the tokens: beyond
#: this (64 tokens of 32 heads of 128 reach it at 65536 positions) a block walks its token's spans itself, which takes
#: none and is slower (64 tokens of 32 heads of 128 over 8 at 16384 positions: 10.1 ms against 1.9).  Recorded graphs keep
#: the buffer that they were recorded with, so the smaller ones it grew from may stay beside it.
MOST_SCRATCH = 256 << 20


def supports(q, pages, head_dim, v_dim, n_q_heads, n_kv_heads) -> bool:
    return (q.dtype == torch.float32 and pages.dtype == torch.float32 and head_dim in HEAD_DIMS and v_dim == head_dim
            and n_q_heads % n_kv_heads == 0 and n_q_heads // n_kv_heads <= MOST_GROUP
            and q.data_ptr() % 16 == 0 and pages.data_ptr() % 16 == 0)


def tiles(q, pages, out, info, n, block_table, n_q_heads, n_kv_heads, head_dim, page_size, window, scale, singles=False):
    """``info`` int32 [n * 4]: the tiles of ``attention_mma.describe_segments`` (``singles``: its single tokens)."""
    lib = core()
    _check(lib, lib.qil_attention_f32_tiles(
        _p(q), _p(pages), _p(out), _p(info), c_int(n), c_int(1 if singles else 0), c_int(attention_mma.QUERY_TILE), _p(block_table),
        c_int(block_table.shape[1]), c_int(n_q_heads), c_int(n_kv_heads), c_int(head_dim), c_int(page_size), c_int(pages.shape[0]),
        c_int(window), c_float(scale), _stream()), "attention_f32 (tiles)")


def singles(q, pages, out, info, n, n_spans, scratch, block_table, n_q_heads, n_kv_heads, head_dim, page_size, window, scale):
    """``info`` int32 [n * 4]: single tokens, every position below ``n_spans * SPAN``.  ``scratch``: (partial sums, their
    (maximum, sum) pairs, tickets) of ``attention_mma.decode_scratch``."""
    part_o, part_ml, tickets = scratch
    if part_o.numel() < n * n_q_heads * n_spans * head_dim or part_ml.numel() < 2 * n * n_q_heads * n_spans \
            or tickets.numel() < n * n_kv_heads:
        raise KernelError("attention_f32: scratch too small")
    lib = core()
    _check(lib, lib.qil_attention_f32_singles(
        _p(q), _p(pages), _p(out), _p(info), c_int(n), c_int(n_spans), _p(part_o), _p(part_ml), _p(tickets), _p(block_table),
        c_int(block_table.shape[1]), c_int(n_q_heads), c_int(n_kv_heads), c_int(head_dim), c_int(page_size), c_int(pages.shape[0]),
        c_int(window), c_float(scale), _stream()), "attention_f32 (single tokens)")


def attend(ctx, q, cache, out, n_q_heads, n_kv_heads, head_dim, window, scale):
    """q float32 [N, Hq*D], out [N, Hq*D]; cache a KVCacheView whose pages already hold this step's keys and values."""
    _need(q, "q", torch.float32, 2); _need(out, "out", torch.float32, 2)
    check_pages(cache.pages, torch.float32, n_kv_heads, cache.page_size, head_dim, head_dim, "attention_f32")
    if q.shape[1] != n_q_heads * head_dim or out.shape != q.shape:
        raise KernelError("attention_f32: q/out shapes do not match the head counts")
    arrays, counts = attention_mma.step_plan(ctx)
    n_tiles, n_single = counts["tile_info"] // 4, counts["decode_info"] // 4
    shape = (cache.block_table, n_q_heads, n_kv_heads, head_dim, cache.page_size, window, scale)
    if n_tiles:
        tiles(q, cache.pages, out, arrays["tile_info"], n_tiles, *shape)
    if n_single:
        n_spans = -(-ctx.max_context // SPAN)
        if n_q_heads // n_kv_heads > MOST_SINGLE_GROUP or 4 * n_single * n_q_heads * n_spans * head_dim > MOST_SCRATCH:
            tiles(q, cache.pages, out, arrays["decode_info"], n_single, *shape, singles=True)
        else:
            scratch = attention_mma.decode_scratch(ctx, n_single, n_q_heads, n_spans, head_dim, most=MOST_SCRATCH)
            singles(q, cache.pages, out, arrays["decode_info"], n_single, n_spans, scratch, *shape)
