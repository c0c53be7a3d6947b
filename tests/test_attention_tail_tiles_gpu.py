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
