"""The bfloat16 norm at the widths where a row's threads change and at row counts that end inside a block, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [8, 96, 1024, 1032, 2048, 2056, 4096, 4104, 8192])
@pytest.mark.parametrize("weight_dtype", [torch.bfloat16, torch.float32])
def test_rmsnorm_of_many_and_few_rows(width, weight_dtype):
    from qwen_inference_lab_b200.kernels import ops
    generator = torch.Generator().manual_seed(width)
    x = torch.randn(601, width, generator=generator).bfloat16().cuda()
    w = (1 + 0.1 * torch.randn(width, generator=generator)).to(weight_dtype).cuda()
    exact = x.double() * (x.double().square().mean(-1, keepdim=True) + 1e-6).rsqrt() * w.double()
    whole = torch.full_like(x, float("nan"))
    ops.rmsnorm(x, w, 1e-6, out=whole)                        # several rows a block, the last block partly empty
    # two roundings to bfloat16, each within 2^-8 of what it rounds (half a step of 8 bits is 2^-9 to 2^-8)
    assert bool(((whole.double() - exact).abs() <= 2.0 ** -7 * 1.01 * exact.abs()).all())
    for n in (1, 3, 592, 593):
        assert torch.equal(ops.rmsnorm(x[:n], w, 1e-6), whole[:n]), n           # a row is the same bits in any company
    rows = torch.tensor([600, 0, 7], dtype=torch.int32).cuda()
    assert torch.equal(ops.rmsnorm(x, w, 1e-6, rows=rows), whole[rows.long()])


def in_the_order_of_256_threads(x, w, eps):
    """The norm in float32 on the CPU: thread t has the vectors of eight t, t + 256, ... and adds their squares one after the other
    (a square of two bfloat16 is exact, so a fused multiply-add rounds as the sum does); the lanes of a warp and then the warps as
    trees."""
    rows, width = x.shape
    f = torch.zeros(rows, 8192)
    f[:, :width] = x.float()
    f = f.view(rows, 4, 256, 8)
    sq = torch.zeros(rows, 256)
    for i in range(4):
        for k in range(8):
            sq = sq + f[:, i, :, k] * f[:, i, :, k]
    sq = sq.view(rows, 8, 32)
    for half in (16, 8, 4, 2, 1):
        sq = sq[..., :half] + sq[..., half:2 * half]
    sq = sq[..., 0]
    for half in (4, 2, 1):
        sq = sq[..., :half] + sq[..., half:2 * half]
    scale = 1.0 / torch.sqrt(sq / width + eps)
    return ((x.float() * scale).bfloat16().float() * w.float()).bfloat16()


@pytest.mark.parametrize("width", [96, 264, 1024, 1032, 2048, 4096, 8192])
@pytest.mark.parametrize("weight_dtype", [torch.bfloat16, torch.float32])
def test_the_sum_of_a_row_has_one_order(width, weight_dtype):
    """Whoever takes a row, a warp or a block, in whatever company: the same bits."""
    from qwen_inference_lab_b200.kernels import ops
    generator = torch.Generator().manual_seed(width + 1)
    x = torch.randn(601, width, generator=generator).bfloat16()
    w = (1 + 0.1 * torch.randn(width, generator=generator)).to(weight_dtype)
    wanted = in_the_order_of_256_threads(x, w, 1e-6)
    for n in (1, 64, 601):
        assert torch.equal(ops.rmsnorm(x[:n].cuda(), w.cuda(), 1e-6).cpu(), wanted[:n]), n
