"""Sets of short and well-anchored patterns alone, which have a stage kernel of their
own, on both sides of 256 tiles (where one launch finishes the search), and the same sets with one pattern of each other kind, against
the oracle."""
import numpy as np
import pytest

import oracle
from oneline_b200 import datagen

pytestmark = pytest.mark.gpu

TILE = 16384
OTHERS = [b"mids!", b"||||||||", b"ZZZZZZZZZ", b"||||||||q"]


@pytest.mark.parametrize("n", [256 * TILE, 256 * TILE + 1, 257 * TILE - 3, 300 * TILE + 77])
@pytest.mark.parametrize("count", [1, 2, 5, 7])
def test_plain_and_mixed_sets(parser, n, count):
    text = np.resize(datagen.corpus(1 << 20, count), n)
    for i, p in enumerate(OTHERS + [b"anchored-and-rare", b"xq"]):
        for at in (5 + 40 * i, 256 * TILE - 30 + 7 * i, n - 40 - 20 * i):
            at = min(at, n - len(p))
            text[at: at + len(p)] = np.frombuffer(p, np.uint8)
    data = text.tobytes()
    plain = [b"anchored-and-rare", b"xq", data[-12:], b"|", data[70_000:70_040], b"- ", data[TILE - 9: TILE + 9]][:count]
    doc = parser.upload(data)
    want = {p: oracle.find_all(data, p) for p in plain + OTHERS}
    for extra in [[]] + [[p] for p in OTHERS]:
        for p, r in zip(plain + extra, parser.search_document_multi(doc, plain + extra, n)):
            assert r.total_matches == len(want[p]) and np.array_equal(r.offsets, want[p]), (p, extra)
