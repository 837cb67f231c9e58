"""Lines whose end lies many 16 KiB tiles away, in texts of more than 1024 tiles:
the next newline in the tiles that one round trip covers, just past them, far
away, in a tile with more lines than a slot holds, in the last tile, or nowhere,
against the oracle; and what such a line costs."""
import numpy as np
import pytest

import oracle
from oneline_b200 import _lib

pytestmark = pytest.mark.gpu

TILE = 16384


@pytest.mark.parametrize("tiles", [1025, 1300, 8200])
def test_end_of_a_long_line(parser, tiles):
    n = tiles * TILE - 5
    ends = [[], [tiles - 1], [1023, 1024], [255, 512, 769], [256, 514], [1, 257 + 1, 1024], [0, 600, 601]]
    ends += [[32 * 32, 32 * 32 + 1], [tiles - 2, tiles - 1]]
    for i, at in enumerate(ends):
        text = np.full(n, ord("y"), np.uint8)
        for t in (t for t in at if t < tiles):
            text[t * TILE + (t * 7919 + i) % (TILE - 8)] = ord("\n")
        if i % 3 == 0:  # a prefix, and an end in "\r"s, that only the whole line shows
            text[:8] = np.frombuffer(b"|| | - i", np.uint8)
            text[n - 3:] = ord("\r")
        if i % 3 == 1 and at and at[-1] < tiles:  # the line ends in a tile with more lines than a slot holds
            text[at[-1] * TILE + 300: at[-1] * TILE + 3300] = ord("\n")
        data = text.tobytes()
        offs, nodes = oracle.parse(data)
        doc = parser.upload(data)
        assert np.array_equal(doc.read_offsets(), offs), at
        assert np.array_equal(doc.read_kinds(), nodes["kind"].astype(np.uint8)), at
        assert np.array_equal(doc.read_nodes(), nodes), at
        doc.free()


def test_one_line_is_not_dearer_than_many(parser):
    """512 MiB that are one line against the same in lines of 64 KiB, whose arrays
    have to be written as well (1.5 times as dear with a scan tile by tile)."""
    import torch

    stream = torch.cuda.ExternalStream(_lib.load().ol_ctx_stream(parser.ctx))

    def parse_ms(text):
        doc = parser.upload(text)
        times = []
        for _ in range(15):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            _lib.check(_lib.load().ol_doc_reparse_async(parser.ctx, doc.handle), parser.ctx)
            b.record(stream)
            b.synchronize()
            times.append(a.elapsed_time(b))
        doc.free()
        return float(np.median(times))

    text = np.full(512 << 20, ord("x"), np.uint8)
    one = parse_ms(text)
    text[::65536] = ord("\n")
    many = parse_ms(text)
    assert one < 1.2 * many, (one, many)
