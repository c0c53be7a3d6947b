"""The crossover points between kernels: measured, not derived, and kept in one place.

Each value says from where on one kernel hands over to another.  They are no limits (a kernel refuses
what it cannot take on its own) and nothing depends on them for correctness; they were measured on one
B200 at the layer sizes named beside them, and another width or another GPU may want others.  Any of
them can be overridden for a process with ``QIL_TUNE_<NAME>=<number>`` (read once, at import) or by
assigning to the attribute before the first step.
"""
from __future__ import annotations

import os


def _tuned(name, default):
    raw = os.environ.get(f"QIL_TUNE_{name}")
    return type(default)(raw) if raw is not None else default


#: Most rows the weight-streaming decode product takes (``gemm_small_m``); the kernel's own limit is 16.
SMALL_M_MAX_ROWS = _tuned("SMALL_M_MAX_ROWS", 16)
#: With 9 to 16 rows the decode product keeps three stages in flight instead of four; on a matrix of at
#: least this many elements it then loses to the library (151936 x 4096 vocabulary head, 16 rows: 274 us
#: against 211 us).
SMALL_M_LIBRARY_ELEMENTS = _tuned("SMALL_M_LIBRARY_ELEMENTS", 1 << 28)
#: With at most 8 rows the decode product gives a block 32 output features instead of 16 when that still leaves
#: this many blocks (one for each of the 148 SMs: 4096 features make 128 and lose, 19.7 -> 22.9 us at K 12288)
#: and the matrix has fewer than this many elements (a stream as long as a vocabulary head's runs 3 % faster on
#: the longer row segments of the 16-feature blocks: 194.7 against 200.9 us).  In between the wider block wins by
#: its fewer instructions per weight byte (6144 x 4096 with the norm: 20.3 -> 18.5 us; 24576 x 4096: 37.2 -> 36.2).
SMALL_M_WIDE_MIN_BLOCKS = _tuned("SMALL_M_WIDE_MIN_BLOCKS", 148)
SMALL_M_WIDE_MAX_ELEMENTS = _tuned("SMALL_M_WIDE_MAX_ELEMENTS", 1 << 28)
#: From this many rows on the gate/up product runs on the tcgen05 kernels (the first row count the decode product does not
#: take): the streaming one up to the limits below, from there on the tile kernel.
TILE_KERNEL_MIN_ROWS = _tuned("TILE_KERNEL_MIN_ROWS", 17)
#: Up to this many rows the streaming tcgen05 kernel (``gemm_tc.gemm_rows``) takes the gate/up product of a matrix of at
#: least 148 tiles of 128 features, and any number up to its 128 of a smaller one (24576 x 4096 against the tile kernel:
#: 38.9 / 41.0 us at 64 rows, 42.9 / 40.3 at 128; 6144 x 1024: 8.2 / 12.3 and 10.0 / 12.3).  Where K is cut over a cluster the
#: sums come in another order than the tile kernel's; against 64 bits both are as far off (12 shapes of K 96 to 25600, 17 to 128
#: rows, 3 seeds each: relative errors of 3.50e-3 to 3.65e-3, ratio 0.996 to 1.003 either way).
ROWS_PAIRS_MAX = _tuned("ROWS_PAIRS_MAX", 64)
#: ... and every other product instead of the library's.  Alone the two are even (4096 x 4096 12.1 / 11.1 us at 32 rows, 4096 x
#: 12288 22.9 / 23.5, 1024 x 2048 6.5 / 7.2); in a chain this one's start is hidden.  A recorded step of the 28-layer 1024-wide
#: model with both, with gate/up alone and without: 1231 / 1252 / 1385 us at 17 rows, 1291 / 1391 / 1510 at 24, 1383 / 1419 / 1538 at
#: 32, 1440 / 1418 / 1457 at 40; of the 36-layer 4096-wide one 3780 / 3871 / 3976, 3851 / 3951 / 4057, 4001 / 4022 / 4122, 4140 / 4073 / 4142.
#: (The kernel itself takes up to 128 rows here too, for whoever raises the line.)  Against 64 bits a plain product is as far
#: off as the library's (1.66e-3), one with a residual less (1.66e-3 against 2.15e-3: one rounding instead of two).
ROWS_PLAIN_MAX = _tuned("ROWS_PLAIN_MAX", 32)
#: From this many rows on the q/k/v product runs on the tcgen05 kernels with its tail fused; below, the pair
#: kernel has too few 256 x 256 tiles for the SM pairs and the library product plus the tail kernel win
#: (6144 x 4096 at 2048 rows: 86 us against 75 + 24 us; at 256 rows the library wins).
QKV_TAIL_MIN_ROWS = _tuned("QKV_TAIL_MIN_ROWS", 512)
#: The single-token attention's cost model, in units of the time a block takes to stream one 64-key tile:
#: a block's start-up (its description, page ids and first tile arrive one after the other) and what each
#: further span adds to the merge.  Fitted to the recorded decode step of 32/8 heads of 128 at a context of
#: 8192 (batch 8: 4.84 ms with 5 or 6 spans, 4.97 with 4, 5.1 with 7 to 9; batch 1 flat from 16 to 43 spans).
SPAN_STARTUP_TILES = _tuned("SPAN_STARTUP_TILES", 2.0)
SPAN_MERGE_TILES = _tuned("SPAN_MERGE_TILES", 0.15)
