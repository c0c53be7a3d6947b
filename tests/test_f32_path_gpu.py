"""The products and the attention of the true 32-bit path at the edges of their kernels' ranges, against 64 bits; a row's
and a token's result is the same bits in whatever company it comes."""
import pytest
import torch

from tests.test_kernels_gpu import attention_case, flat_meta

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(7, 4), (64, 96), (65, 132), (200, 1024), (1000, 3080), (9000, 260), (50000, 64), (120, 256)])
@pytest.mark.parametrize("full", [False, True], ids=["plain", "epilogue"])
def test_gemm_f32_rows(n, k, full):
    from qwen_inference_lab_b200.kernels import ops
    generator = torch.Generator().manual_seed(n + k)
    draw = lambda *shape: torch.randn(*shape, generator=generator).cuda()
    a, w = draw(300, k), draw(n, k) * 0.1
    bias, scale, residual = (draw(n), draw(n), draw(300, n)) if full else (None, None, None)
    exact = a.double() @ w.double().t()
    # a chain of k / 16 products, 16 such sums and three operations of the epilogue; up to 256 products one chain
    bound = ((k / 16 if k > 256 else k) + 20) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t())
    if full:
        exact, bound = exact + bias.double(), bound + 2.0 ** -22 * bias.double().abs()
        exact, bound = exact * scale.double(), bound * scale.double().abs()
        exact, bound = exact + residual.double(), bound + 2.0 ** -22 * (exact.abs() + residual.double().abs())
    whole = None
    for m in (300, 1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 129):
        rest = residual[:m].clone() if full else None
        out = rest if full else torch.full((m, n), float("nan"), device="cuda")        # the residual may be the output
        ops.gemm_f32(a[:m], w, bias=bias, residual=rest, out=out, col_scale=scale)
        assert bool(((out.double() - exact[:m]).abs() <= bound[:m]).all()), m
        whole = out if whole is None else whole
        assert torch.equal(out, whole[:m]), m


CASES = [
    # n_q, n_kv, d, lengths, chunk starts, page, window
    (4, 2, 128, [1, 255, 256, 257, 512, 513, 700], [0, 254, 0, 200, 511, 300, 699], 16, 0),
    (6, 2, 32, [65, 3, 511, 1], [64, 0, 300, 0], 3, 0),
    (3, 3, 64, [64, 65, 1025], [63, 0, 1000], 8, 0),
    (8, 1, 64, [300, 129, 700], [250, 128, 699], 16, 100),
    (16, 1, 128, [600, 70], [500, 69], 32, 0),
    (64, 1, 32, [270], [200], 16, 300),
]


@pytest.mark.parametrize("case", CASES, ids=[f"case{i}" for i in range(len(CASES))])
def test_attention_f32(case):
    from qwen_inference_lab_b200.kernels import attention_f32, ops
    n_q, n_kv, d, lengths, starts, page, window = case
    q, pool, table, meta, expected = attention_case(n_q, n_kv, d, lengths, starts, torch.float32, page, seed=5, window=window)
    q, pool, table = q.cuda(), pool.cuda(), table.cuda()
    as_int = lambda values: torch.tensor(values, dtype=torch.int32).cuda()
    shape = (table, n_q, n_kv, d, page, window, d ** -0.5)
    tile_info, single_info, at = [], [], 0
    for start, length, pos0, row in zip(meta["seg_start"], meta["seg_len"], meta["seg_pos0"], meta["seg_row"]):
        for off in range(0, length, 64):
            tile_info += [start + off, pos0 + off, min(64, length - off), row]
        single_info += [v for j in range(length) for v in (start + j, pos0 + j, row, 0)]
    tiled, alone = torch.full_like(q, float("nan")), torch.full_like(q, float("nan"))
    attention_f32.tiles(q, pool, tiled, as_int(tile_info), len(tile_info) // 4, *shape)
    n = len(single_info) // 4
    if n_q // n_kv <= attention_f32.MOST_SINGLE_GROUP:
        n_spans = (max(lengths) + 255) // 256 + 1                  # one spare span
        scratch = (torch.full((n * n_q * n_spans * d,), float("nan"), device="cuda"),
                   torch.full((n * n_q * n_spans * 2,), float("nan"), device="cuda"),
                   torch.zeros(n * n_kv, dtype=torch.int32, device="cuda"))
        attention_f32.singles(q, pool, alone, as_int(single_info), n, n_spans, scratch, *shape)
        assert int(scratch[2].abs().max()) == 0
        assert torch.equal(alone, tiled)
    walked = torch.full_like(q, float("nan"))
    attention_f32.tiles(q, pool, walked, as_int(single_info), n, *shape, singles=True)
    assert torch.equal(walked, tiled)
    torch.testing.assert_close(tiled.cpu(), expected.float(), atol=2e-6, rtol=2e-5)
    generic = torch.empty_like(q)
    positions, token_row = flat_meta(meta)
    ops.attention_generic(q, pool, generic, positions, token_row, table, n_q, n_kv, d, page, window, d ** -0.5)
    torch.testing.assert_close(tiled, generic, atol=2e-6, rtol=2e-5)


def both_kernels(q, pool, table, info, n_q, n_kv, d, page, window=0):
    """The same tokens (first, position, row) through the tile kernel, the span kernel and the general one."""
    from qwen_inference_lab_b200.kernels import attention_f32, ops
    as_int = lambda values: torch.tensor(values, dtype=torch.int32).cuda()
    shape = (table, n_q, n_kv, d, page, window, d ** -0.5)
    tiled, alone, generic = (torch.full_like(q, 7.0) for _ in range(3))
    n, n_spans = len(info), max(pos for _, pos, _ in info) // 256 + 1
    attention_f32.tiles(q, pool, tiled, as_int([v for at, pos, row in info for v in (at, pos, 1, row)]), n, *shape)
    scratch = (torch.empty(n * n_q * n_spans * d, device="cuda"), torch.empty(n * n_q * n_spans * 2, device="cuda"),
               torch.zeros(n * n_kv, dtype=torch.int32, device="cuda"))
    attention_f32.singles(q, pool, alone, as_int([v for at, pos, row in info for v in (at, pos, row, 0)]), n, n_spans, scratch, *shape)
    ops.attention_generic(q, pool, generic, as_int([pos for _, pos, _ in info]), as_int([row for _, _, row in info]), *shape)
    return tiled, alone, generic


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")], ids=["nan", "inf", "minus_inf"])
@pytest.mark.parametrize("place", ["key", "value"])
def test_attention_f32_of_what_is_no_number(place, bad):
    """A key or a value that is not finite: seen, it shows as in the general kernel (a key alone in its span too); unseen
    (behind the token, before the window, in an unused slot), it does not."""
    n_q, n_kv, d, page, length = 4, 2, 64, 16, 600
    generator = torch.Generator().manual_seed(8)
    pool = torch.randn(length // page + 1, 2, n_kv, page, d, generator=generator)
    at = 512                                             # the first key of the third span
    column = slice(None) if place == "key" and bad != bad else 0
    pool[at // page, 0 if place == "key" else 1, :, at % page, column] = bad
    table = torch.arange(length // page + 1, dtype=torch.int32).view(1, -1).cuda()
    positions = [10, 255, 511, 512, 513, 599]
    q = torch.randn(len(positions), n_q * d, generator=generator).cuda()
    for window in (0, 90, 1):
        tiled, alone, generic = both_kernels(q, pool.cuda(), table, [(i, pos, 0) for i, pos in enumerate(positions)], n_q, n_kv, d, page, window)
        torch.testing.assert_close(tiled, generic, atol=2e-6, rtol=2e-5, equal_nan=True)
        torch.testing.assert_close(alone, tiled, atol=0.0, rtol=0.0, equal_nan=True)
        for i, pos in enumerate(positions):
            seen = at <= pos and not (window and pos - window + 1 > at)
            assert seen or bool(torch.isfinite(tiled[i]).all())


def test_a_refused_launch_leaves_no_error_behind():
    """A product on a stream whose recording has been broken fails on the host; the next kernel does not answer for it."""
    from qwen_inference_lab_b200.kernels import ops
    from qwen_inference_lab_b200.kernels.ops import KernelError
    a, w, x, gain = (torch.ones(*shape, device="cuda") for shape in ((4, 512), (64, 512), (3, 64), (64,)))
    out, normed = torch.empty(4, 64, device="cuda"), torch.empty(3, 64, device="cuda")
    ops.gemm_f32(a, w, out=out)
    ops.rmsnorm(x, gain, 1e-6, out=normed)
    torch.cuda.synchronize()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="thread_local")
        with pytest.raises(RuntimeError):
            stream.synchronize()                               # not while it records: the recording is broken from here on
        with pytest.raises(KernelError):
            ops.gemm_f32(a, w, out=out)
        with pytest.raises(RuntimeError):
            graph.capture_end()
    ops.rmsnorm(x, gain, 1e-6, out=normed)
    torch.testing.assert_close(normed, torch.ones_like(normed))
