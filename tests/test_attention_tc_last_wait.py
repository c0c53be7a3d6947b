"""The tcgen05 attention's last wait: a warp of softmax rows that never rescales may be two tiles ahead of one that does."""
import itertools

import pytest
import torch


def read_too_early(n_tiles, rescaling, wait_on_last_tile):
    """The barrier protocol between one warp that never rescales (A), one that rescales at the tiles ``rescaling`` (B) and
    the MMA warp, walked through every order of their steps.  The barrier of the second MMAs shows the parity of its
    phase alone: a wait for parity p passes when the phase before the current one has it.  True if A can read the output
    before the last second MMA is done."""
    def program(tiles):
        steps = []
        for j in range(n_tiles):
            steps.append(("scores", j))
            if j > 0 and (j in tiles or (wait_on_last_tile and j == n_tiles - 1)):
                steps.append(("output", j - 1))
            steps.append(("publish", j))
        return steps + [("output", n_tiles - 1), ("read", None)]
    programs = (program(()), program(rescaling))
    seen, todo = set(), [(0, 0, 0)]                       # steps done by A and B, second MMAs done
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        at, done = state[:2], state[2]
        published = [sum(kind == "publish" for kind, _ in programs[w][:at[w]]) for w in (0, 1)]
        if done < min(published):                         # a second MMA needs every warp's P
            todo.append((*at, done + 1))
        for w in (0, 1):
            if at[w] == len(programs[w]):
                continue
            kind, j = programs[w][at[w]]
            if kind == "scores" and done < j - 1:         # scores j are issued behind second MMA j - 2
                continue
            if kind == "output" and (done - 1) & 1 != j & 1:
                continue
            if kind == "read" and done < n_tiles:
                return True
            todo.append((at[0] + (w == 0), at[1] + (w == 1), done))
    end = (len(programs[0]), len(programs[1]), n_tiles)
    assert end in seen                                    # and nobody waits for good
    return False


@pytest.mark.parametrize("n_tiles", range(1, 7))
def test_no_order_of_steps_reads_the_output_early(n_tiles):
    for count in range(n_tiles):
        for rescaling in itertools.combinations(range(1, n_tiles), count):
            assert not read_too_early(n_tiles, rescaling, wait_on_last_tile=True)
            if n_tiles > 1:
                assert read_too_early(n_tiles, rescaling, wait_on_last_tile=False)     # what the wait is for


@pytest.mark.gpu
@pytest.mark.parametrize("length", [192, 256, 384, 448])
@pytest.mark.parametrize("quarter", range(4))
def test_one_warp_rescales_at_the_tile_before_the_last(length, quarter):
    """A key that stands out for 32 of a tile's 128 queries, in the key tile before the last: their warp rescales there and is
    late, the others are not."""
    from qwen_inference_lab_b200.kernels import attention_tc
    from tests.plain import qwen3_plain as plain
    generator = torch.Generator().manual_seed(length + quarter)
    n_q, n_kv, d, page, requests = 32, 8, 128, 16, 6
    start, per = length - 128, length // page
    pool = torch.zeros(requests * per, 2, n_kv, page, d, dtype=torch.bfloat16)
    q, expected = [], []
    for r in range(requests):
        keys, values, queries = (torch.randn(length, heads, d, generator=generator) for heads in (n_kv, n_kv, n_q))
        keys[:, :, 0] = 0.0
        queries[:, :, 0] = 0.0
        keys[length - 128, :, 0] = 40.0                  # its score: 40 * 12 / sqrt(128) = 42, in units of log2 61
        queries[start + 32 * quarter:start + 32 * quarter + 32, :, 0] = 12.0
        keys, values, queries = keys.bfloat16(), values.bfloat16(), queries.bfloat16()
        pool[r * per:(r + 1) * per, 0] = keys.view(per, page, n_kv, d).transpose(1, 2)
        pool[r * per:(r + 1) * per, 1] = values.view(per, page, n_kv, d).transpose(1, 2)
        full = plain.causal_attention(queries.float(), keys.float(), values.float(), d ** -0.5)
        q.append(queries[start:].reshape(128, n_q * d))
        expected.append(full[start:].reshape(128, n_q * d))
    table = torch.arange(requests * per, dtype=torch.int32).view(requests, per).cuda()
    info = torch.tensor([v for r in range(requests) for v in (128 * r, start, 128, r)], dtype=torch.int32).cuda()
    q, pool = torch.cat(q).cuda(), pool.cuda()
    out = torch.empty_like(q)
    for _ in range(3):
        out.fill_(float("nan"))
        attention_tc.prefill(q, pool, out, info, requests, table, n_q, n_kv, page, d ** -0.5, head_dim=d)
        attention_tc.check()
        torch.testing.assert_close(out.float().cpu(), torch.cat(expected), atol=1.6e-2, rtol=8e-3)
