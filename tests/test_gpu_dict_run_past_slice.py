"""Runs that cover a slice's last position and end up to 65 positions past it: the
hits of patterns that end in them, against the oracle, and no walk for a run whose
end no pattern that starts in the slice can reach (63 positions and more)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

SLICE = 256  # of a text this short
N = 4 * SLICE


@pytest.mark.parametrize("before", [1, 3, 70])
def test_run_ends_past_a_slice(parser, before):
    pats = [b"|" * r + b"x" for r in (3, 4, 10, 60, 61, 62, 63)] + [b"|" * r + b"xy" for r in (3, 61, 62)]
    pats += [b"|" * k for k in (4, 5, 62, 63, 64)]
    ps = parser.compile_patterns(None, pats)
    walked = {}
    for past in (2, 3, 4, 30, 60, 61, 62, 63, 64, 65):
        text = np.full(N, ord("y"), np.uint8)
        text[2 * SLICE - before: 2 * SLICE + past] = ord("|")
        text[2 * SLICE + past] = ord("x")
        counts, hp, ho, total = oracle.CpuBaseline(threads=1).many(pats).find_all_par(text.tobytes())
        r = parser.search_many(parser.upload(text), ps, 4096)
        assert r.total_hits == total and np.array_equal(r.counts, counts), past
        assert np.array_equal(r.hits["pattern"], hp) and np.array_equal(r.hits["offset"], ho), past
        walked[past] = parser.dict_stats()["walked"]
    # the run's end is walked in its own slice, and once more for the starts before it
    assert all(walked[p] == walked[64] + 1 for p in (3, 4, 30, 60, 61, 62)), walked
    assert walked[63] == walked[64] == walked[65], walked
