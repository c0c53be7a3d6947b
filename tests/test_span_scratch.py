"""The partial sums of the single-token attention: how the buffer grows, and what is done beyond its limit."""
from types import SimpleNamespace

import pytest
import torch

from qwen_inference_lab_b200.kernels import attention_f32, attention_mma


def sizes(requests, most):
    ctx, found = SimpleNamespace(extras={}, device=torch.device("cpu")), []
    for slots in requests:
        found.append(attention_mma.decode_scratch(ctx, slots, 4, 2, 32, most=most)[0].numel())
    return found


def test_the_buffer_doubles_up_to_the_limit_and_not_beyond():
    unit = 4 * 2 * 32                                            # values a token
    assert sizes((1, 2, 3, 5, 9), None) == [unit, 2 * unit, 4 * unit, 8 * unit, 16 * unit]
    assert sizes((1, 2, 3, 5, 9, 10), 4 * 10 * unit) == [unit, 2 * unit, 4 * unit, 8 * unit, 10 * unit, 10 * unit]
    assert sizes((8, 9), 4 * 10 * unit)[-1] == 10 * unit        # not 16


def test_the_float32_attention_hands_its_limit_on(monkeypatch):
    asked = []
    monkeypatch.setattr(attention_mma, "decode_scratch", lambda ctx, *shape, **more: asked.append(more))
    monkeypatch.setattr(attention_f32, "_need", lambda *a: None)
    monkeypatch.setattr(attention_f32, "check_pages", lambda *a: None)
    monkeypatch.setattr(attention_f32, "singles", lambda *a: asked.append("spans"))
    monkeypatch.setattr(attention_f32, "tiles", lambda *a, singles=False: asked.append("walked"))
    plan = SimpleNamespace(array={"tile_info": None, "decode_info": None}, count={"tile_info": 0, "decode_info": 4 * 3})
    ctx = SimpleNamespace(plans={attention_mma.PLAN_KEY: plan}, max_context=1000)
    q = torch.empty(3, 4 * 32)
    cache = SimpleNamespace(pages=None, block_table=None, page_size=16)
    need = 4 * 3 * 4 * 4 * 32                                    # four spans
    for limit, expected in ((need, [{"most": need}, "spans"]), (need - 1, ["walked"])):
        asked.clear()
        monkeypatch.setattr(attention_f32, "MOST_SCRATCH", limit)
        attention_f32.attend(ctx, q, cache, torch.empty_like(q), 4, 2, 32, 0, 1.0)
        assert asked == expected


@pytest.mark.gpu
def test_both_sides_of_the_limit_give_the_same_bits(monkeypatch):
    n_q, n_kv, d, page, length, n = 8, 4, 64, 16, 1400, 5
    torch.manual_seed(4)
    per = -(-length // page)
    cache = SimpleNamespace(pages=torch.randn(n * per, 2, n_kv, page, d).cuda(), page_size=page,
                            block_table=torch.arange(n * per, dtype=torch.int32).view(n, per).cuda())
    info = [v for i in range(n) for v in (i, length - 1 - 250 * i, i, length)]
    plan = SimpleNamespace(array={"tile_info": None, "decode_info": torch.tensor(info, dtype=torch.int32).cuda()},
                           count={"tile_info": 0, "decode_info": len(info)})
    ctx = SimpleNamespace(plans={attention_mma.PLAN_KEY: plan}, max_context=length, extras={}, device=torch.device("cuda"))
    q = torch.randn(n, n_q * d).cuda()
    out = [torch.full_like(q, float("nan")) for _ in range(2)]
    attention_f32.attend(ctx, q, cache, out[0], n_q, n_kv, d, 0, d ** -0.5)
    assert ctx.extras
    monkeypatch.setattr(attention_f32, "MOST_SCRATCH", 1)
    ctx.extras = {}
    attention_f32.attend(ctx, q, cache, out[1], n_q, n_kv, d, 0, d ** -0.5)
    assert not ctx.extras and torch.equal(*out) and bool(torch.isfinite(out[0]).all())
