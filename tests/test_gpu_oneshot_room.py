"""A one-shot parse whose caller has room for too few lines does no work for the
results that it cannot write: as many launches as one that only counts."""
import ctypes

import numpy as np
import pytest

from oneline_b200 import NODE_DTYPE, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tail", [b"", b"\n"])
@pytest.mark.parametrize("n", [4000, 300_001])  # through one scratch buffer, and through a document's own
def test_room_too_small_costs_no_nodes(parser, n, tail):
    L = _lib.load()
    text = np.frombuffer((b"| an entry\n" * n)[: n - 1] + (tail or b"x"), np.uint8)
    lines = int(np.count_nonzero(text == 10)) + (not tail)
    offs, nodes, cnt = np.full(lines, 7, np.uint32), np.zeros(lines, NODE_DTYPE), ctypes.c_uint64()

    def launches(nodes_to, cap):
        before = L.ol_launch_count()
        _lib.check(L.ol_parse_raw(parser.ctx, text.ctypes.data, n, offs.ctypes.data, nodes_to, cap, ctypes.byref(cnt)),
                   parser.ctx)
        assert cnt.value == lines
        return L.ol_launch_count() - before

    count_only = launches(None, 0)
    assert launches(nodes.ctypes.data, lines - 2) == count_only and np.all(offs == 7)
    launches(nodes.ctypes.data, lines - 1)  # (a final newline starts no line: known only after the parse)
    assert np.all(offs == 7)
    assert launches(nodes.ctypes.data, 2**64 - 1) > count_only and nodes["kind"].all()
