"""The products of the true 32-bit path at the edges of their kernels' ranges, against 64 bits; a row's result is the same
bits in whatever company it comes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(7, 4), (64, 96), (65, 132), (200, 1024), (1000, 3080), (9000, 260), (50000, 64)])
@pytest.mark.parametrize("full", [False, True], ids=["plain", "epilogue"])
def test_gemm_f32_rows(n, k, full):
    from qwen_inference_lab_b200.kernels import ops
    generator = torch.Generator().manual_seed(n + k)
    draw = lambda *shape: torch.randn(*shape, generator=generator).cuda()
    a, w = draw(300, k), draw(n, k) * 0.1
    bias, scale, residual = (draw(n), draw(n), draw(300, n)) if full else (None, None, None)
    exact = a.double() @ w.double().t()
    # a chain of k / 16 products, 16 such sums and three operations of the epilogue
    bound = (k / 16 + 20) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t())
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
