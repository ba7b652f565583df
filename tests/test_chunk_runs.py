"""Which requests of a step run as chunks (`ops.chunk_runs`), on the host."""
import random

import pytest

from tensorline_b200.ops import channel_chunks, chunk_runs


@pytest.mark.parametrize("seed", range(20))
def test_runs_of_random_steps(seed):
    r = random.Random(seed)
    lens = [r.choice([0, 1, 1, r.randint(2, 40), r.randint(40, 700)]) for _ in range(r.randint(1, 12))]
    chunk, least = r.choice([32, 64]), r.choice([1, 16, 32, 96])
    start = [sum(lens[:i]) for i in range(len(lens) + 1)]
    words, n_rows, n_runs, n_firsts, longest = chunk_runs(start, chunk, least)
    want_rows, want_runs, want_firsts = [], [], []
    for b, n in enumerate(lens):
        if n == 0:
            continue
        if n < least:
            want_runs.append([b, 0, 0, 0])
            continue
        first, count = len(want_rows), -(-n // chunk)
        want_firsts.append(first)
        want_runs.append([b, first, count, 0])
        want_rows += [[b, c, count, first] for c in range(count)]
    assert (n_rows, n_runs, n_firsts) == (len(want_rows), len(want_runs), len(want_firsts))
    assert words.tolist() == [x for r in want_rows + want_runs for x in r] + want_firsts
    assert longest == max([n for n in lens if n < least], default=0)
    if least == 1:
        assert want_rows == channel_chunks(start, chunk)[0].tolist()
