"""Which kernel takes a bfloat16 product's rows: the rule over all forms it looks at, and what the parts then compute."""
import pytest
import torch

from qwen_inference_lab_b200.kernels import gemm_tc, ops
from qwen_inference_lab_b200.parts.feed_forward import GatedMLP
from qwen_inference_lab_b200.parts.linear import Linear


def matrix(rows, columns, dtype=torch.bfloat16):
    return torch.empty(rows, columns, dtype=dtype)


def off_by(tensor, elements):
    """The same values in storage that starts ``elements`` off a 16-byte boundary."""
    storage = torch.empty(tensor.numel() + elements + 8, dtype=tensor.dtype, device=tensor.device)
    first = (-storage.data_ptr() // tensor.element_size()) % 8 + elements
    return storage[first:first + tensor.numel()].view(tensor.shape).copy_(tensor)


LARGE, SMALL = 148 * 128, 148 * 128 - 16        # rows of a gate/up matrix on both sides of the rule's line


def test_rows_that_the_streaming_kernel_takes():
    for m in range(1, 140):
        x = matrix(m, 64)
        assert gemm_tc.rows_usable(x, matrix(96, 64)) == (17 <= m <= 32)
        assert gemm_tc.rows_usable(x, matrix(LARGE, 64), silu_pairs=True) == (17 <= m <= 64)
        assert gemm_tc.rows_usable(x, matrix(SMALL, 64), silu_pairs=True) == (17 <= m <= 128)


def test_forms_that_it_does_not_take():
    x, w, good = matrix(20, 64), matrix(96, 64), matrix(20, 96)
    assert gemm_tc.rows_usable(x, w, residual=good, out=matrix(20, 96)) and gemm_tc.rows_usable(x, w, residual=good, out=good)
    assert not gemm_tc.rows_usable(x.float(), w) and not gemm_tc.rows_usable(x, w.float())
    assert not gemm_tc.rows_usable(matrix(20, 60), matrix(96, 60))                         # rows that end off 16 bytes
    assert not gemm_tc.rows_usable(x, matrix(100, 64))
    assert not gemm_tc.rows_usable(matrix(64, 20).t(), w) and not gemm_tc.rows_usable(matrix(20, 128)[:, :64], w)
    assert not gemm_tc.rows_usable(x, matrix(64, 96).t()) and not gemm_tc.rows_usable(x, matrix(96, 128)[:, :64])
    assert not gemm_tc.rows_usable(off_by(x, 1), w) and not gemm_tc.rows_usable(x, off_by(w, 4))
    for name in ("residual", "out"):
        for bad in (off_by(good, 1), off_by(good, 4), matrix(96, 20).t(), matrix(20, 192)[:, ::2], matrix(20, 200)[:, :96]):
            assert not gemm_tc.rows_usable(x, w, **{name: bad}), name


@pytest.fixture
def chosen(monkeypatch):
    """The names of the bfloat16 products that were called, in their order."""
    names = []
    for module, name in ((gemm_tc, "gemm_rows"), (gemm_tc, "gemm_tc"), (ops, "gemm_small_m"), (torch, "mm"), (torch, "addmm")):
        def noted(*args, _call=getattr(module, name), _name=name, **more):
            names.append(_name)
            return _call(*args, **more)
        monkeypatch.setattr(module, name, noted)
    return names


def draw(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).bfloat16().cuda()


@pytest.mark.gpu
@pytest.mark.parametrize("bias", [False, True], ids=["plain", "bias"])
@pytest.mark.parametrize("form", ["new", "in_place", "strided_out", "unaligned_residual", "unaligned_both"])
def test_linear_at_the_rules_edges(chosen, bias, form):
    k, n = 128, 144
    linear = Linear(k, n, name="x", bias=bias)
    linear.weight.data = draw(n, k, scale=k ** -0.5)
    if bias:
        linear.bias.data = draw(n, seed=1)
    linear.finalize("cuda", torch.bfloat16)
    for m in (16, 17, 32, 33):
        x, residual = draw(m, k, seed=m), draw(m, n, seed=m + 100)
        raw = x.double() @ linear.weight.data.double().t()
        product = raw + (linear.bias.data.double() if bias else 0.0)
        fits = m <= 16 or form in ("new", "in_place")
        if m <= 16 and form not in ("new", "in_place"):
            continue                                              # the decode product's own conditions are older
        chosen.clear()
        if form == "new":
            expected, out = product, linear.forward(None, x)
        elif form == "strided_out":
            wide = draw(m, 2 * n)
            expected, out = product, linear.forward(None, x, out=wide[:, :n])
        else:
            expected = product + residual.double()
            residual = off_by(residual, 1) if form != "in_place" else residual
            out = linear.forward(None, x, residual=residual, out=off_by(residual, 3) if form == "unaligned_both" else residual)
        assert (chosen[0] == "gemm_small_m") == (m <= 16) and (chosen[0] == "gemm_rows") == (17 <= m <= 32 and fits), (m, chosen)
        # rounded to bfloat16 up to three times: the product, the product with the bias, both with the residual, each within
        # 2^-8 of what it rounds
        bound = 2.0 ** -8 * (raw.abs() + product.abs() + expected.abs()) * 1.01 + 1e-4
        assert bool(((out.double() - expected).abs() <= bound).all()), (m, form)


@pytest.mark.gpu
@pytest.mark.parametrize("inner", [SMALL // 2, LARGE // 2])
def test_gated_mlp_at_the_rules_edges(chosen, inner):
    hidden = 64
    mlp = GatedMLP(hidden, inner, names=dict(gate="g", up="u", down="d"))
    gate, up, down = draw(inner, hidden, scale=0.2), draw(inner, hidden, seed=1, scale=0.2), draw(hidden, inner, seed=2, scale=inner ** -0.5)
    mlp.gate_up.parts_w[0].data, mlp.gate_up.parts_w[1].data, mlp.down.weight.data = gate, up, down
    mlp.finalize("cuda", torch.bfloat16)
    assert mlp.pairs8
    most = 64 if 2 * inner >= LARGE else 128
    for m in (16, 17, 32, 33, 64, 65, 128, 129):
        x, residual = draw(m, hidden, seed=m), draw(m, hidden, seed=m + 100)
        chosen.clear()
        out = mlp.forward(None, x, residual=residual.clone())
        first = "gemm_small_m" if m <= 16 else "gemm_rows" if m <= most else "gemm_tc"
        second = "gemm_small_m" if m <= 16 else "gemm_rows" if m <= 32 else "addmm"
        assert chosen == [first, second], (m, chosen)
        inside = torch.nn.functional.silu(x.double() @ gate.double().t()) * (x.double() @ up.double().t())
        expected = inside @ down.double().t() + residual.double()
        # the hidden values carry three roundings of 2^-8, whose errors add up over the down product; two more at the end
        slack = 3 * 2.0 ** -8 * (inside.abs() @ down.double().t().abs())
        assert bool(((out.double() - expected).abs() <= slack + 2.0 ** -7 * (expected.abs() + residual.double().abs())).all()), m
