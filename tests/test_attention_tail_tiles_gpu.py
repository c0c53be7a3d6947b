"""Tiles of fewer than 128 tokens through the tcgen05 attention, and the rule that makes them."""
import numpy as np
import pytest
import torch

from tests.test_kernels_gpu import attention_case, close

CASES = [
    # n_q, n_kv, d, lengths, chunk starts, page, window
    (4, 2, 128, [1, 2, 129, 200, 66], [0, 0, 1, 73, 1], 16, 0),
    (8, 2, 128, [1024, 300, 65], [897, 299, 0], 8, 0),
    (6, 1, 128, [700, 128, 64], [637, 1, 1], 64, 0),
    (4, 4, 64, [513, 255], [450, 128], 32, 100),
    (2, 1, 16, [400, 70], [333, 3], 16, 0),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=[f"case{i}" for i in range(len(CASES))])
def test_tiles_of_fewer_tokens(case):
    from qwen_inference_lab_b200.kernels import attention_tc
    n_q, n_kv, d, lengths, starts, page, window = case
    q, pool, table, meta, expected = attention_case(n_q, n_kv, d, lengths, starts, torch.bfloat16, page, seed=31, window=window)
    info = []
    for start, length, pos0, row in zip(meta["seg_start"], meta["seg_len"], meta["seg_pos0"], meta["seg_row"]):
        for off in range(0, length, 128):
            info += [start + off, pos0 + off, min(128, length - off), row]
    out = torch.full(q.shape, float("nan"), dtype=torch.bfloat16).cuda()
    attention_tc.prefill(q.cuda(), pool.cuda(), out, torch.tensor(info, dtype=torch.int32).cuda(), len(info) // 4,
                         table.cuda(), n_q, n_kv, page, d ** -0.5, window=window, head_dim=d)
    torch.cuda.synchronize()
    attention_tc.check()
    close(out, expected, torch.bfloat16, scale=2)      # no row is left out, none written for another


def test_every_token_is_in_one_tile():
    from qwen_inference_lab_b200.kernels import attention_mma
    lens = np.array([2, 64, 65, 128, 129, 192, 193, 300, 5, 1, 20])
    starts = np.array([0, 0, 0, 0, 0, 0, 0, 0, 255, 7, 200])
    first = np.concatenate([[0], lens.cumsum()[:-1]])
    plan = attention_mma.describe_segments(first, starts, lens, np.arange(len(lens)))
    seen = np.zeros(lens.sum(), dtype=int)
    for name, most in (("big_tile_info", 128), ("rest_tile_info", 64)):
        for token, pos, count, row in plan[name].reshape(-1, 4):
            assert 0 < count <= most and pos - starts[row] == token - first[row]
            seen[token:token + count] += 1
            tail = lens[row] % 128
            if name == "rest_tile_info":       # whole tiles never, tails up to 64 tokens of a short context only
                assert token - first[row] >= lens[row] - tail and tail <= 64 and starts[row] + lens[row] <= attention_mma.TAIL_CONTEXT
    for token, _, _, _ in plan["decode_info"].reshape(-1, 4):
        seen[token] += 1
    assert (seen == 1).all()


@pytest.mark.gpu
@pytest.mark.parametrize("d,length,start", [(128, 700, 663), (128, 1500, 1391), (64, 900, 898), (32, 400, 335)])
def test_a_tail_is_as_exact_as_in_the_64_token_kernel(d, length, start):
    # which kernel takes a segment's tail is a matter of time alone: the error of its tiles may not be larger.  Both round
    # the weights and the result to bfloat16 at the same places, so the errors of some 10^5 values agree to a per cent
    from qwen_inference_lab_b200.kernels import attention_mma, attention_tc
    q, pool, table, meta, expected = attention_case(16, 4, d, [length, length + 64], [start, start + 64], torch.bfloat16, 16, seed=3)
    q, pool, table = q.cuda(), pool.cuda(), table.cuda()
    def tiles(size):
        info = [v for first, n, pos0, row in zip(meta["seg_start"], meta["seg_len"], meta["seg_pos0"], meta["seg_row"])
                for off in range(0, n, size) for v in (first + off, pos0 + off, min(size, n - off), row)]
        return torch.tensor(info, dtype=torch.int32).cuda(), len(info) // 4
    by_64, by_128 = torch.empty_like(q), torch.empty_like(q)
    attention_mma.prefill(q, pool, by_64, *tiles(64), table, 16, 4, d, 16, 0, d ** -0.5)
    attention_tc.prefill(q, pool, by_128, *tiles(128), table, 16, 4, 16, d ** -0.5, head_dim=d)
    error = lambda out: float((out.cpu().double() - expected.double()).norm() / expected.double().norm())
    assert error(by_128) <= 1.01 * error(by_64)
    attention_tc.check()


OPTIONS = {
    # d, v_dim, window, and what else the scores get
    "slopes": (64, 64, 0, dict(slopes=True)),
    "cap": (128, 128, 0, dict(softcap=4.0)),
    "cap_and_slopes": (32, 32, 0, dict(softcap=3.0, slopes=True)),
    "chunk": (64, 64, 0, dict(chunk=150)),
    "sink": (128, 128, 0, dict(sink=True)),
    "chunk_cap_sink": (64, 64, 0, dict(chunk=96, softcap=5.0, sink=True)),
    "window_and_slopes": (64, 64, 90, dict(slopes=True)),
    "wide_values": (16, 64, 0, dict()),
    "narrow_values": (128, 64, 0, dict(sink=True)),
    "values_window": (48, 80, 70, dict(slopes=True)),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", OPTIONS)
def test_tiles_of_fewer_tokens_with_every_score_option(name):
    """Tails of 1 to 127 tokens behind contexts in and out of step with key tiles and chunks, unused slots full of NaN, beside
    the general kernel (float32 arithmetic on the same bfloat16 operands)."""
    from qwen_inference_lab_b200.kernels import attention_tc, ops
    d, v_dim, window, options = OPTIONS[name]
    n_q, n_kv, page = 8, 2, 16
    segments = [(0, 1), (63, 2), (64, 127), (149, 65), (300, 37), (511, 3), (700, 100)]          # (position, tokens)
    generator = torch.Generator().manual_seed(sum(map(ord, name)))
    draw = lambda *shape: torch.randn(*shape, generator=generator)
    pages, table = [], torch.full((len(segments), 60), -1, dtype=torch.int32)
    for row, (start, count) in enumerate(segments):
        for at in range(0, start + count, page):
            keys, values = draw(n_kv, page, d), draw(n_kv, page, v_dim)
            keys[:, max(0, start + count - at):] = values[:, max(0, start + count - at):] = float("nan")
            table[row, at // page] = len(pages)
            pages.append(torch.cat([keys.reshape(-1), values.reshape(-1)]))
    pages = torch.stack(pages).bfloat16().cuda()
    if v_dim == d:
        pages = pages.view(-1, 2, n_kv, page, d)
    table = table.cuda()
    q = draw(sum(count for _, count in segments), n_q * d).bfloat16().cuda()
    info, positions, rows = [], [], []
    for row, (start, count) in enumerate(segments):
        info += [len(positions), start, count, row]
        positions += range(start, start + count)
        rows += [row] * count
    as_int = lambda values: torch.tensor(values, dtype=torch.int32).cuda()
    slopes = (0.02 * torch.arange(1, n_q + 1)).cuda() if options.get("slopes") else None
    sinks = draw(n_q).cuda() if options.get("sink") else None
    softcap, chunk = options.get("softcap", 0.0), options.get("chunk", 0)
    log2e = 1.4426950408889634
    out = torch.full((q.shape[0], n_q * v_dim), float("nan"), dtype=torch.bfloat16, device="cuda")
    attention_tc.prefill(q, pages, out, as_int(info), len(segments), table, n_q, n_kv, page, d ** -0.5,
                         slopes_log2=None if slopes is None else slopes * log2e, chunk=chunk,
                         sink_log2=None if sinks is None else sinks * log2e, softcap=softcap, window=window, head_dim=d, v_dim=v_dim)
    attention_tc.check()
    expected = torch.empty_like(out)
    ops.attention_generic(q, pages, expected, as_int(positions), as_int(rows), table, n_q, n_kv, d, page, window, d ** -0.5,
                          v_dim=v_dim, slopes=slopes, softcap=softcap, chunk=chunk, sink_logits=sinks)
    close(out, expected.float(), torch.bfloat16, scale=2)
