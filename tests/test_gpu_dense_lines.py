"""Texts of more than 1024 tiles in which nearly every byte ends a line (many tiles
with more lines than a slot holds, and some without), against the oracle; and what
such a text costs."""
import numpy as np
import pytest

import oracle
from oneline_b200 import _lib

pytestmark = pytest.mark.gpu

TILE = 16384


@pytest.mark.parametrize("line", [b"\n", b"|\n", b"|a\n", b"\n\n\n |x\n"])
@pytest.mark.parametrize("tiles", [1025, 1777])
def test_dense_tiles(parser, line, tiles):
    n = tiles * TILE - 100
    text = np.resize(np.frombuffer(line, np.uint8), n)
    for t in range(5, tiles - 2, 7):  # every seventh tile is one line and a part of the next tile's
        text[t * TILE + 900: (t + 1) * TILE + t % 700] = ord("y")
    data = text.tobytes()
    offs, nodes = oracle.parse(data)
    doc = parser.upload(data)
    assert np.array_equal(doc.read_offsets(), offs)
    assert np.array_equal(doc.read_kinds(), nodes["kind"].astype(np.uint8))
    assert np.array_equal(doc.read_nodes(), nodes)


def test_cost_of_empty_lines(parser):
    import torch

    stream = torch.cuda.ExternalStream(_lib.load().ol_ctx_stream(parser.ctx))

    def parse_ms(line):
        doc = parser.upload(np.resize(np.frombuffer(line, np.uint8), 32 << 20))
        times = []
        for _ in range(25):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            _lib.check(_lib.load().ol_doc_reparse_async(parser.ctx, doc.handle), parser.ctx)
            b.record(stream)
            b.synchronize()
            times.append(a.elapsed_time(b))
        doc.free()
        return float(np.median(times))

    # 8 times as many tile rounds and 300 times as many lines: 10 times the time, 13 with idle SMs
    assert parse_ms(b"\n") < 11.4 * parse_ms(b"a" * 299 + b"\n")
