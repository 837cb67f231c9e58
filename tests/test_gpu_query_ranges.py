"""Node queries over ranges that begin and end anywhere, results around the size
that comes back in one copy, depths past the clamped array, and more blocks than
add up the counts themselves, against the oracle's nodes."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def text_of(n: int, deepest: int) -> bytes:
    rng = np.random.default_rng(n)
    depth = np.abs(np.cumsum(rng.integers(-2, 3, n))) % 6
    depth[n // 3] = deepest
    kinds = [b"", b" x", b" =h", b" @e", b" - i", b" :c", b" -. o", b" // c"]
    pick = rng.integers(0, len(kinds), n)
    return b"".join(b"|" * int(d) + kinds[int(k)] + b"\n" for d, k in zip(depth, pick))


def want(nodes, lo, hi, kind, depth):
    m = np.ones(hi - lo, bool)
    if kind:
        m &= nodes["kind"][lo:hi] == kind
    if depth is not None:
        m &= nodes["depth"][lo:hi] == depth
    return (np.nonzero(m)[0] + lo).astype(np.uint32)


@pytest.mark.parametrize("deepest", [7, 254, 255, 300])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 4095, 4097, 70_001])
def test_ranges(parser, n, deepest):
    text = text_of(n, deepest)
    _, nodes = oracle.parse(text)
    ends = oracle.full_tree(nodes)["subtree_end"]
    doc = parser.upload(text)
    tree = parser.build_tree(doc, strict_depth=False)
    roots = sorted({0, n - 1, n // 3, n // 2, min(5, n - 1), int(np.argmax(ends - np.arange(n)))})
    for kind, depth in [(None, None), (4, None), (None, 2), (1, 0), (7, 3), (None, deepest), (2, 254), (None, 255), (9, None), (300, 1)]:
        w = want(nodes, 0, n, kind, depth)
        for room in (0, 1, 16383, 16384, 16385, n):
            r = parser.query_document(doc, kind, depth, room)
            assert r.total_matches == w.size and np.array_equal(r.indices, w[:room]), (kind, depth, room)
        for root in roots:
            w = want(nodes, root, int(ends[root]), kind, depth)
            r = parser.query_subtree(doc, tree, root, kind, depth, n)
            assert r.total_matches == w.size and np.array_equal(r.indices, w), (root, kind, depth)


def test_many_blocks(parser):
    n = 8193 * 4096 + 5
    text = np.full(n, ord("\n"), np.uint8)  # blank lines, and a few that are not
    at = np.arange(7, n - 1, 40_009)
    text[at] = ord("x")
    doc = parser.upload(text.tobytes())
    _, nodes = oracle.parse(text.tobytes())
    w = want(nodes, 0, len(nodes), 1, None)
    r = parser.query_document(doc, 1, None, 100_000)
    assert r.total_matches == w.size and np.array_equal(r.indices, w)
    r = parser.query_document(doc, None, 0, 20_000)
    assert r.total_matches == len(nodes) and np.array_equal(r.indices, np.arange(20_000))
