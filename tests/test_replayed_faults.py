"""A replayed step reports what its kernels found, as the step that recorded it does."""
import pytest
import torch

from qwen_inference_lab_b200.kernels import ops


def test_marks_collects_every_word_once_and_ends_with_its_block():
    words = [ops.ErrorWord(str) for _ in range(3)]
    with ops.marks() as outer:
        words[0].mark()
        with ops.marks() as inner:
            words[1].mark(); words[1].mark()
        words[0].mark()
    words[2].mark()
    assert outer == words[:2] and inner == words[1:2]
    with pytest.raises(KeyError):
        with ops.marks() as broken:
            raise KeyError
    words[0].mark()
    assert broken == []


@pytest.mark.gpu
@pytest.mark.parametrize("wait", [True, False], ids=["waiting", "running_ahead"])
def test_a_replay_is_checked(tmp_path, wait):
    from qwen_inference_lab_b200.engine import StepEntry
    from qwen_inference_lab_b200.kernels import gemm_tc
    from tests import harness
    from tests.tiny_configs import TINY_D
    harness.write_folder(TINY_D, 3, tmp_path)
    rows = gemm_tc.MIN_ROWS + 3                              # more than the decode product takes
    model, cache, runner = harness.build_engine_parts(tmp_path, torch.bfloat16, num_pages=2 * rows, page_size=16, max_requests=rows)
    for i in range(rows):
        cache.admit(i)
    step = lambda: runner.run([StepEntry(i, [i + 1], [0]) for i in range(rows)])
    step()                                                   # records
    runner.check()
    step()
    runner.check()
    word = gemm_tc.error_word(model.device)
    runner.check()
    word.fill_(4)                                            # what a wait that ran out in a replayed kernel leaves there
    late = 0
    with pytest.raises(ops.KernelError, match="code 4"):
        for late in range(ops.ErrorWord.REPLAYS + 2):        # running ahead: when enough replays have passed, one check late
            step()
            torch.cuda.synchronize()
            runner.check(wait)
    assert late == (0 if wait else ops.ErrorWord.REPLAYS)
    step()
    runner.check()
