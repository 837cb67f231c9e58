"""Subtree queries in documents of many lines: the passes cover the subtree, not
the document, past the number of blocks at which its end is read first (4096, of
4096 lines each, from the root on), and the answer is the same on both sides."""
import numpy as np
import pytest

from oneline_b200 import _lib

pytestmark = pytest.mark.gpu

BLOCK = 4096


@pytest.mark.parametrize("blocks,more", [(4096, 0), (4096, 1), (8193, 5)])
def test_small_subtree_of_many_lines(parser, blocks, more):
    n = blocks * BLOCK + more
    text = np.tile(np.frombuffer(b"a\n", np.uint8), n)
    kids = [(5, 1), (21, 3000), (40_000, 1)]  # line, lines of its subtree after it
    parts, at = [], 0
    for line, k in kids:
        parts += [text[2 * at: 2 * (line + 1)], np.frombuffer(b"|@\n" * k, np.uint8)]
        at = line + 1 + k
    parts.append(text[2 * at:])
    doc = parser.upload(np.concatenate(parts))
    assert doc.line_count() == n
    tree = parser.build_tree(doc)
    for line, k in kids + [(0, 0), (n - 1, 0)]:
        before = _lib.load().ol_launch_count()
        r = parser.query_subtree(doc, tree, line, 3, None, 10_000)
        launches = _lib.load().ol_launch_count() - before
        assert r.total_matches == k and np.array_equal(r.indices, np.arange(line + 1, line + 1 + k))
        assert launches == 2, "the counts of a few blocks take no scan of their own"
    r = parser.query_subtree(doc, tree, 0, None, 0, 10)  # its first line only
    assert r.total_matches == 1 and r.indices.tolist() == [0]
