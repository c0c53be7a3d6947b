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
#: least 148 tiles of 128 features, and any number up to its 128 of a smaller one (us, alone, against the tile kernels, the even
#: tiles among them: 24576 x 4096 37.0 / 39.9 at 33 rows, 38.1 / 40.1 at 64, 41.0 / 40.3 at 96, 42.4 / 40.4 at 128; 6144 x 1024
#: 5.9 / 7.9, 6.8 / 7.9, 8.4 / 8.0, 9.0 / 8.5: the line of the smaller one was drawn before there were even tiles).  Where K is cut
#: over a cluster the
#: sums come in another order than the tile kernel's; against 64 bits both are as far off (12 shapes of K 96 to 25600, 17 to 128
#: rows, 3 seeds each: relative errors of 3.50e-3 to 3.65e-3, ratio 0.996 to 1.003 either way).
ROWS_PAIRS_MAX = _tuned("ROWS_PAIRS_MAX", 64)
#: ... and every other product instead of the library's.  Alone the two are even (us, this one / the library's: 4096 x 4096
#: 10.3 / 9.4 at 32 rows, 4096 x 12288 20.5 / 21.4, 1024 x 3072 5.9 / 7.4, 4096 x 1024 5.1 / 4.5); in a chain this one's start is
#: hidden.  A recorded step of the 28-layer 1024-wide model behind 500 cached tokens with both, with gate/up alone and without (us):
#: 1170 / 1358 / 1323 at 17 rows, 1284 / 1433 / 1471 at 24, 1367 / 1384 / 1491 at 32, 1447 / 1540 / 1566 at 40, 1544 / 1593 / 1619 at 48,
#: 1976 / 2033 / 2063 at 64; of the 36-layer 4096-wide one 3662 / 3918 / 4054, 3813 / 4019 / 4158, 3992 / 4074 / 4201, 4155 / 4247 / 4331,
#: 4218 / 4324 / 4404, 4885 / 4844 / 4917.  So the line could lie at 48 now; it is where it was before the kernel's issue got cheaper
#: (it lost at 40 then), and a step's bits with it.
#: (The kernel itself takes up to 128 rows here too, for whoever raises the line.)  Against 64 bits a plain product is as far
#: off as the library's (1.66e-3), one with a residual less (1.66e-3 against 2.15e-3: one rounding instead of two).
ROWS_PLAIN_MAX = _tuned("ROWS_PLAIN_MAX", 32)
#: From this many rows on the q/k/v product runs on the tcgen05 kernels with its tail fused; below, the library's product
#: and the tail kernel.  us, fused / apart: 6144 x 4096 at 256 rows 24 / 20, 512 30 / 28, 700 33 / 34, 1021 46 / 46, 2048 77 / 90,
#: 2920 105 / 138; 4096 x 1024 at 512 17.2 / 12.0, 700 17.8 / 14.2, 1021 17.8 / 17.8, 2048 28.6 / 29.9, 2920 33.9 / 40.0.  (Kernels alone,
#: recorded: in a step that is not, as prompts are, the host launches one kernel less.)
QKV_TAIL_MIN_ROWS = _tuned("QKV_TAIL_MIN_ROWS", 512)
#: The single-token attention's cost model, in units of the time a block takes to stream one 64-key tile:
#: a block's start-up (its description, page ids and first tile arrive one after the other) and what each
#: further span adds to the merge.  Fitted to the recorded decode step of 32/8 heads of 128 at a context of
#: 8192 (batch 8: 4.84 ms with 5 or 6 spans, 4.97 with 4, 5.1 with 7 to 9; batch 1 flat from 16 to 43 spans).
SPAN_STARTUP_TILES = _tuned("SPAN_STARTUP_TILES", 2.0)
SPAN_MERGE_TILES = _tuned("SPAN_MERGE_TILES", 0.15)
