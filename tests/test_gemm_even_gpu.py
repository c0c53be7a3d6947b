"""The tcgen05 product whose tiles cut the tokens evenly: every epilogue at the edges of tiles, against 64 bits and the other kernels."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def draw(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).bfloat16().cuda()


@pytest.mark.parametrize("tokens", [16, 32, 48, 176, 256])
@pytest.mark.parametrize("m,n,k", [(1, 8, 8), (31, 136, 64), (177, 264, 72), (521, 640, 448), (1030, 1040, 384)])
def test_tiles_of_any_number_of_tokens(m, n, k, tokens):
    from qwen_inference_lab_b200.kernels import gemm_tc
    a, w, bias, residual = draw(m, k), draw(n, k, seed=1, scale=k ** -0.5), draw(n, seed=2), draw(m, n, seed=3)
    raw = a.double() @ w.double().t()
    wanted = raw + bias.double() + residual.double()
    # float32 sums and one rounding to bfloat16 (half a step of 8 bits)
    bound = 2.0 ** -8 * 1.01 * wanted.abs() + (k + 4) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t() + 8)
    out = residual.clone()
    gemm_tc.gemm_tc(a, w, bias=bias, residual=out, out=out, tile_tokens=tokens)
    assert bool(((out.double() - wanted).abs() <= bound).all())
    gemm_tc.check()


@pytest.mark.parametrize("tokens", [16, 48, 176, 256])
@pytest.mark.parametrize("m,n,k", [(1, 16, 8), (31, 144, 72), (177, 272, 200), (521, 640, 448), (1030, 1040, 384)])
def test_gate_and_up_in_one(m, n, k, tokens):
    from qwen_inference_lab_b200.kernels import gemm_tc, ops
    a, w = draw(m, k), draw(n, k, seed=1, scale=2 * k ** -0.5)
    fused = gemm_tc.gemm_tc(a, w, silu_pairs=True, tile_tokens=tokens).double()
    gate, up = (a.double() @ w.double().t()).view(m, n // 16, 2, 8).unbind(2)
    slack = (k + 4) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t()).view(m, n // 16, 2, 8)
    # the sums in float32, then rounded to bfloat16 (half a step of 8 bits); silu's slope is at most 1.1
    half = 2.0 ** -8 * 1.01
    off_gate, off_up = half * gate.abs() + slack[:, :, 0], half * up.abs() + slack[:, :, 1]
    silu = torch.nn.functional.silu(gate)
    off_silu = 1.1 * off_gate
    off_silu += half * (silu.abs() + off_silu)
    wanted = silu * up
    off = off_silu * (up.abs() + off_up) + silu.abs() * off_up
    off += half * (wanted.abs() + off)
    assert bool(((fused.view_as(wanted) - wanted).abs() <= off).all())
    # and beside the same product with its activation apart, which does not divide approximately
    hidden = ops.silu_mul(gemm_tc.gemm_tc(a, w, tile_tokens=tokens), pairs8=True).double()
    assert bool(((fused - hidden).abs() <= 2.0 ** -6 * hidden.abs()).all())
    gemm_tc.check()


@pytest.mark.parametrize("m,n,k", [(255, 9216, 96), (1021, 6144, 1024), (700, 4608, 768)])
def test_gate_and_up_have_the_bits_of_the_other_kernels(m, n, k):
    """Products that the rule leaves to the tile and pair kernels."""
    from qwen_inference_lab_b200.kernels import gemm_tc
    from tests.test_even_rule import taken
    a, w = draw(m, k), draw(n, k, seed=1, scale=k ** -0.5)
    assert taken(m, n, k) == 0
    wanted = gemm_tc.gemm_tc(a, w, silu_pairs=True)
    for tokens in (16, 96, 176, 256):
        assert torch.equal(gemm_tc.gemm_tc(a, w, silu_pairs=True, tile_tokens=tokens), wanted), tokens
    gemm_tc.check()


@pytest.mark.parametrize("m,n_q,n_kv,page,bias,norms,rope", [(300, 3, 1, 8, True, True, True), (521, 4, 2, 16, False, True, True),
                                                             (260, 2, 0, 16, False, False, False), (200, 4, 2, 8, True, True, True),
                                                             (700, 32, 8, 16, False, True, True)])
def test_the_tail_of_the_projection(m, n_q, n_kv, page, bias, norms, rope):
    """The bits of the kernels with one token a lane, which take these as the rule has it: a token's queries and keys do not depend
    on the tiles that a step's size picks."""
    from qwen_inference_lab_b200.kernels import gemm_tc
    from qwen_inference_lab_b200.parts.rotary import rotary_table
    heads, k = n_q + 2 * n_kv, 256
    a, w, b = draw(m, k), draw(heads * 128, k, seed=1, scale=0.1), draw(heads * 128, seed=2) if bias else None
    q_norm, k_norm = ((1 + 0.3 * draw(128, seed=s)).bfloat16() if norms else None for s in (3, 4))
    table = rotary_table(128, 10000.0, 600, torch.bfloat16).cuda() if rope else None
    first = m // 3                             # two requests; the table has no entry for the last tokens of the second
    positions = torch.cat([torch.arange(5, 5 + first), torch.arange(m - first)]).int().cuda()
    token_row = torch.cat([torch.ones(first), torch.zeros(m - first)]).int().cuda()
    per = (m - first) // page
    block_table = torch.randperm(2 * per, generator=torch.Generator().manual_seed(5)).int().view(2, per).cuda()
    results = []
    for tokens in (0, 16, 96, 176, 256):
        q = torch.full((m, n_q * 128), 7.0, dtype=torch.bfloat16, device="cuda")
        pages = torch.full((2 * per, 2, max(n_kv, 1), page, 128), 7.0, dtype=torch.bfloat16, device="cuda")
        gemm_tc.gemm_tc_qkv(a, w, b, q, pages if n_kv else None, table, q_norm, k_norm, 1e-5, positions, token_row, block_table, n_q, n_kv,
                            page, tile_tokens=tokens)
        gemm_tc.check()
        results.append((q, pages))
    for q, pages in results[1:]:
        for got, wanted in ((q, results[0][0]), (pages, results[0][1])):
            assert torch.equal(got, wanted)


def test_products_whose_tiles_the_rule_chooses():
    """Whole and ragged numbers of tokens against 64 bits; which kernel takes them is `test_even_rule`'s."""
    from qwen_inference_lab_b200.kernels import gemm_tc
    w = draw(2048, 2048, scale=2048 ** -0.5)
    for m in (129, 255, 256, 257, 300, 512, 521):
        a = draw(m, 2048, seed=m)
        wanted = a.double() @ w.double().t()
        got = gemm_tc.gemm_tc(a, w)
        assert bool(((got.double() - wanted).abs() <= 2.0 ** -8 * 1.01 * wanted.abs() + 2100 * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t())).all())
    gemm_tc.check()


@pytest.mark.parametrize("m,n,k,tokens", [(300, 2048, 1024, 160), (521, 4096, 2048, 0)])
def test_a_weight_that_the_kernel_before_has_just_written(m, n, k, tokens):
    """The norm lets the next kernel begin before it has written its rows."""
    from qwen_inference_lab_b200.kernels import gemm_tc, ops
    a, source, gain = draw(m, k), draw(n, k, seed=1), draw(k, seed=2)
    w = ops.rmsnorm(source, gain, 1e-6)
    torch.cuda.synchronize()
    wanted = gemm_tc.gemm_tc(a, w, tile_tokens=tokens)
    for _ in range(20):
        w.zero_()
        ops.rmsnorm(source, gain, 1e-6, out=w)
        assert torch.equal(gemm_tc.gemm_tc(a, w, tile_tokens=tokens), wanted)
    gemm_tc.check()
