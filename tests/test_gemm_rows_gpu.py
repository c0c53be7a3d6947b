"""The tcgen05 product for a few dozen rows: every width of its accumulator, ragged features and K, K cut over clusters."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def draw(m, n, k):
    generator = torch.Generator().manual_seed(m + 7 * n + 13 * k)
    a = torch.randn(m, k, generator=generator).bfloat16().cuda()
    return a, (torch.randn(n, k, generator=generator) * k ** -0.5).bfloat16().cuda()


@pytest.mark.parametrize("n,k", [(8, 8), (136, 72), (1000, 64), (128, 448), (264, 1024), (4096, 768), (40, 12288), (19208, 200)])
def test_rows(n, k):
    from qwen_inference_lab_b200.kernels import gemm_tc
    for m in (1, 17, 31, 32, 33, 64, 65, 127, 128):
        a, w = draw(m, n, k)
        bias, residual = torch.randn(n).bfloat16().cuda(), torch.randn(m, n).bfloat16().cuda()
        product = a.double() @ w.double().t()
        # float32 sums of k products, then one rounding to bfloat16 (2^-8); with bias and residual two float32 additions more
        slack = (k + 8) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t())
        out = gemm_tc.gemm_rows(a, w, out=torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda"))
        assert bool(((out.double() - product).abs() <= 2.0 ** -8 * product.abs() + slack + 1e-30).all()), m
        whole = product + bias.double() + residual.double()
        slack += 2.0 ** -22 * (product.abs() + bias.double().abs() + residual.double().abs())
        gemm_tc.gemm_rows(a, w, bias=bias, residual=residual, out=residual)         # in place
        assert bool(((residual.double() - whole).abs() <= 2.0 ** -8 * whole.abs() + slack).all()), m
        again = gemm_tc.gemm_rows(a, w)
        assert torch.equal(again, out)                                              # the same bits on every launch
    gemm_tc.check()


@pytest.mark.parametrize("n,k", [(16, 8), (144, 72), (6144, 512), (19216, 136)])
def test_rows_of_gate_and_up(n, k):
    from qwen_inference_lab_b200.kernels import gemm_tc
    for m in (17, 32, 33, 64, 100, 128):
        a, w = draw(m, n, k)
        out = gemm_tc.gemm_rows(a, w, silu_pairs=True)
        product = (a.double() @ w.double().t()).view(m, n // 16, 2, 8)
        gate, up = product[:, :, 0].reshape(m, -1), product[:, :, 1].reshape(m, -1)
        expected = torch.nn.functional.silu(gate) * up
        # gate, up, silu(gate) and the result are each rounded to bfloat16: four times 2^-8, and |silu'| <= 1.1
        bound = 2.0 ** -8 * (1.1 * gate.abs() * up.abs() + 3.1 * expected.abs()) + 1e-5
        assert bool(((out.double() - expected).abs() <= bound * 1.05).all()), m
    gemm_tc.check()


def test_what_the_rows_kernel_refuses():
    from qwen_inference_lab_b200.kernels import gemm_tc
    from qwen_inference_lab_b200.kernels.ops import KernelError
    a, w = draw(129, 64, 64)
    with pytest.raises(KernelError):
        gemm_tc.gemm_rows(a, w)
    with pytest.raises(KernelError):
        gemm_tc.gemm_rows(a[:20, :60].contiguous(), w[:, :60].contiguous())
    with pytest.raises(KernelError):
        gemm_tc.gemm_rows(a[:20], w[:20], residual=torch.zeros(20, 10, dtype=torch.bfloat16, device="cuda"), silu_pairs=True)
