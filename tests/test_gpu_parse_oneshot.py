"""One-shot parses: texts of up to 256 KiB through one scratch buffer and one
read-back, larger ones and ones with too many lines for it through a document's
own buffers; line counts above and below the first guess, against the oracle."""
import numpy as np
import pytest

import oracle
from oneline_b200 import _lib

pytestmark = pytest.mark.gpu

SHORT = 256 << 10


def text_of(kind: str, n: int) -> bytes:
    part = {"prose": b"|| - an entry of some length, as most lines are\n| =[ A heading ]\r\n\n",
            "dense": b"|a\n",                           # more lines than one in sixteen bytes
            "newlines": b"\n",
            "long": b"||| @" + b"y" * 20000 + b"\n"}[kind]
    return (part * (n // len(part) + 1))[:n]


@pytest.mark.parametrize("kind", ["prose", "dense", "newlines", "long"])
@pytest.mark.parametrize("n", [1, 63, 4099, 16384, SHORT - 1, SHORT, SHORT + 1, (1 << 20) + 1])
def test_one_shot(parser, kind, n):
    text = text_of(kind, n)
    assert len(text) == n
    offs, nodes = oracle.parse(text)
    for given in (text, np.frombuffer(text, np.uint8)):
        tree = parser.parse_raw(given)
        assert np.array_equal(tree.line_offsets, offs)
        for f in nodes.dtype.names:
            assert np.array_equal(tree.nodes[f], nodes[f]), f
    assert np.array_equal(parser.scan_line_offsets(text), offs)


@pytest.mark.parametrize("n", [4099, SHORT + 1])
def test_room_too_small_writes_nothing(parser, n):
    import ctypes

    text = np.frombuffer(text_of("prose", n), np.uint8)
    lines = len(oracle.scan_line_offsets(text.tobytes()))
    out, cnt = np.full(lines, 7, np.uint32), ctypes.c_uint64()
    _lib.check(_lib.load().ol_scan_line_offsets(parser._ctx, text.ctypes.data, n, out.ctypes.data, lines - 1,
                                                ctypes.byref(cnt)), parser._ctx)
    assert cnt.value == lines and np.all(out == 7)
