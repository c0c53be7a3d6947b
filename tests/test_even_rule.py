"""Which products the tcgen05 kernel with evenly cut tokens takes, as its rule says: both sides of every line, with 74 pairs of blocks."""
import re

import pytest

from qwen_inference_lab_b200.kernels import gemm_tc


def taken(m, n, k, tail=False):
    """Tokens a tile, 0 where another kernel takes the product."""
    return gemm_tc.library().qil_gemm_tc_even_tokens(m, n, k, int(tail), 74, 148)


@pytest.mark.parametrize("m,n,k,tokens", [
    (129, 24576, 4096, 144), (300, 24576, 4096, 160), (521, 24576, 4096, 176), (1021, 24576, 4096, 0), (2048, 24576, 4096, 0),
    (255, 24576, 4096, 0), (256, 24576, 4096, 0),                                   # whole tiles of either size
    (300, 12288, 2048, 112), (521, 12288, 2048, 176), (521, 9216, 1536, 0), (700, 9216, 1024, 0),       # more than a wave: a K of 2048
    (129, 6144, 1024, 48), (300, 6144, 1024, 112), (521, 6144, 1024, 176), (560, 6144, 1024, 0), (2920, 6144, 1024, 0),
    (480, 4608, 768, 128), (700, 4608, 768, 0), (300, 4608, 256, 80), (480, 4608, 256, 0), (128, 6144, 96, 48), (255, 6144, 96, 0),
])
def test_gate_and_up(m, n, k, tokens):
    assert taken(m, n, k) == tokens


@pytest.mark.parametrize("m,n,k,tokens", [
    (521, 6144, 4096, 176), (700, 6144, 4096, 0), (776, 6144, 4096, 144), (1021, 6144, 4096, 176), (1500, 6144, 4096, 0),
    (512, 4096, 2048, 128), (600, 4096, 2048, 160), (700, 4096, 2048, 0), (1200, 4096, 2048, 0), (512, 6144, 2560, 176), (560, 6144, 2560, 0),
    (850, 5120, 3072, 128), (1021, 5120, 3072, 0), (1350, 4096, 3584, 160), (1500, 4096, 3584, 0), (1500, 4096, 4096, 176),
    (521, 4096, 1024, 0), (2920, 4096, 1024, 0), (521, 2048, 1536, 0),
])
def test_queries_keys_and_values(m, n, k, tokens):
    assert taken(m, n, k, tail=True) == tokens


def test_tiles_are_what_the_kernel_takes():
    for n, k in ((8, 8), (96, 64), (6144, 1024), (24576, 4096), (151936, 4096)):
        for m in (*range(1, 600, 7), 1021, 2048, 2920, 100000, 1 << 30):
            for tail in (False, True):
                tokens = taken(m, n, k, tail)
                assert tokens % 16 == 0 and 0 <= tokens <= 256


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(129, 2048, 2048), (300, 2048, 2048), (521, 2048, 2048), (700, 4608, 768), (2048, 2048, 768)])
def test_a_call_goes_where_the_rule_says(m, n, k, tmp_path):
    """The call without a tile size launches the even kernel where the rule names one, and another where it does not."""
    import torch
    a, w = (torch.randn(*shape, generator=torch.Generator().manual_seed(1)).bfloat16().cuda() for shape in ((m, k), (n, k)))
    expected = gemm_tc.gemm_tc(a, w)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)                 # its text names the kernels
    graph.enable_debug_mode()
    with torch.cuda.graph(graph):
        got = gemm_tc.gemm_tc(a, w)
    graph.replay()
    torch.cuda.synchronize()
    graph.debug_dump(str(tmp_path / "launches"))
    names = set(re.findall(r"gemm_tc_(?:even_|pair_|rows_)?kernel", (tmp_path / "launches").read_text()))
    tokens = taken(m, n, k)
    assert names == {"gemm_tc_even_kernel" if tokens else "gemm_tc_kernel" if m < 256 else "gemm_tc_pair_kernel"}
    assert torch.equal(got, expected)
    if tokens:
        assert torch.equal(got, gemm_tc.gemm_tc(a, w, tile_tokens=tokens))
    gemm_tc.check()
