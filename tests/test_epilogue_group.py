"""Behind a bounded wait goes on together what meets again without a limit: the lanes of a warp, and the four warps of an even
kernel's epilogue group."""
import itertools
import re
from pathlib import Path

import pytest

from tests.test_chained_waits import KERNELS, SOURCE, block, roles_of

ATTENTION = (Path(__file__).resolve().parent.parent / "qwen_inference_lab_b200" / "csrc" / "attention_tc.cu").read_text()


def outcome(passes, chunks, agree):
    """What becomes of a group whose warp w gets through its wait for tile t if ``passes[t][w]``: (does everybody leave, tiles stored
    by a warp although the wait of one of the group had run out).  ``agree``: they meet behind the wait and leave
    together, else a warp whose wait ran out leaves after its tile."""
    def program(w):
        for t, passed in enumerate(passes):
            if agree:
                yield ("vote", passed[w])
                if not all(passed):
                    return
            for chunk in range(chunks):
                if not agree or chunk > 0:
                    yield ("meet", None)
                yield ("meet", None)
                stored.add((t, w))
            if not passed[w]:
                return
    stored = set()
    programs = [program(w) for w in range(4)]
    at = [next(p, None) for p in programs]
    while any(step is not None for step in at):
        if any(step is None for step in at):
            return False, stored                # three wait for the one that has left
        assert len({kind for kind, _ in at}) == 1
        at = [next(p, None) for p in programs]
    return True, {(t, w) for t, w in stored if not all(passes[t])}


@pytest.mark.parametrize("chunks", [0, 1, 2, 4])
def test_a_wait_that_runs_out_takes_the_group_along(chunks):
    each = list(itertools.product((True, False), repeat=4))
    for passes in itertools.product(each, repeat=2):
        assert outcome(passes, chunks, agree=True) == (True, set())
    if chunks:                                   # what the vote is for
        assert outcome(((True, True, False, True), (True,) * 4), chunks, agree=False)[0] is False
        assert outcome(((False,) * 4,), chunks, agree=False)[1]


def test_the_kernel_votes_before_it_reads_or_stores():
    source = re.sub(r"//[^\n]*", "", SOURCE)
    definition = re.search(r"__global__[^;{]*?\bgemm_tc_even_kernel\(", source)
    body, _ = block(source, source.index(")", definition.end()))
    loop, _ = block(body, body.rindex("for (int tile = pair;"))
    before, after = loop.split("te_group_agrees(group, ok))", 1)
    assert re.search(r"const bool ok = warp_mbar_wait\(&sh->acc_full\[acc\], acc_phase\);", before)
    assert re.search(r"if \(!ok && lane == 0\) atomicExch\(error_word, 5\);\s*if \(!$", before)
    assert re.match(r"\s*break;", after)
    for name in ("te_group_sync", "tmem_load_32", "te_store_rows", "mbar_arrive_cluster"):
        assert name not in before and name in after
    assert "mbar_wait(" not in after
    assert re.search(r"bar\.red\.and\.pred p, %1, 128, q;", SOURCE)


@pytest.mark.parametrize("kernel", KERNELS + ("attn_tc_kernel",))
def test_the_lanes_of_a_warp_go_on_together(kernel):
    """A lane that gave up by itself would be missing from the warp's reads of tensor memory."""
    if kernel == "attn_tc_kernel":
        source = re.sub(r"//[^\n]*", "", ATTENTION)
        role, _ = block(source, source.index("} else if (warp < AT_VALUE_WARP) {") + 2)
    else:
        role = roles_of(kernel)[2]
    waits = re.findall(r"\w*mbar_wait\(", role)
    assert waits and set(waits) == {"warp_mbar_wait("}
