"""Kernels that are launched chained begin while the kernel before them still runs: how long that takes may not count
against their bounded waits."""
import re
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parent.parent / "qwen_inference_lab_b200" / "csrc" / "gemm_tc.cu").read_text()
KERNELS = ("gemm_tc_kernel", "gemm_tc_pair_kernel", "gemm_tc_even_kernel", "gemm_tc_rows_kernel")


def block(text, at):
    """The text between the brace at or after ``at`` and its partner, and where it ends."""
    begin = text.index("{", at)
    depth = 0
    for i in range(begin, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[begin + 1:i], i + 1
    raise AssertionError("unbalanced braces")


def roles_of(kernel):
    """The text of the kernel's three roles: loads, MMAs, epilogue."""
    source = re.sub(r"//[^\n]*", "", SOURCE)
    definition = re.search(r"__global__[^;{]*?\b%s\(" % kernel, source)
    assert re.search(r"qil_launch_(chained|clusters)\(%s\b" % kernel, source)
    body, _ = block(source, source.index(")", definition.end()))
    at, roles = body.index("if (warp == 0) {"), []
    while True:
        role, end = block(body, at)
        roles.append(role)
        follows = re.match(r"\s*else\b", body[end:])
        if not follows:
            break
        at = end
    assert len(roles) == 3
    return roles


@pytest.mark.parametrize("kernel", KERNELS)
def test_every_role_waits_for_the_kernel_before_ahead_of_its_first_bounded_wait(kernel):
    for role in roles_of(kernel):
        assert "mbar_wait(" in role
        assert role.split("mbar_wait(")[0].count("qil_wait_for_producer();") == 1, role[:200]


@pytest.mark.parametrize("kernel", KERNELS)
def test_what_is_copied_ahead_of_the_wait(kernel):
    """The tile kernels take any caller's matrices, the output of the kernel before among them; the streaming one asks for its
    weights first and says so."""
    ahead, after = roles_of(kernel)[0].split("qil_wait_for_producer();")
    copied = re.findall(r"tma_load_2d\w*\([^;]*?&(map_\w+)", ahead)
    assert copied == (["map_w"] if kernel == "gemm_tc_rows_kernel" else [])
    assert "&map_w" in after
