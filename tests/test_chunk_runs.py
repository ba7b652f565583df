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
    rows, runs, firsts, longest = chunk_runs(start, chunk, least)
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
    assert rows.tolist() == want_rows and runs.tolist() == want_runs and firsts.tolist() == want_firsts
    assert longest == max([n for n in lens if n < least], default=0)
    if least == 1:
        assert rows.tolist() == channel_chunks(start, chunk)[0].tolist()
