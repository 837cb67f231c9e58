"""Patterns that are found by their rarest four bytes (all but a few bytes of them
are one common byte): the rare byte at every place, at the text's beginning and
end and around tile edges, against the oracle; and what one costs in a text of the
common byte."""
import numpy as np
import pytest

import oracle
from oneline_b200 import _lib

pytestmark = pytest.mark.gpu

TILE = 16384


def patterns():
    for m in (8, 9, 17, 64, 250, 300, 4097):
        for at in sorted({0, 1, 2, 3, 4, 7, m // 2, m - 5, m - 2, m - 1}):
            for rare in (b"q", b" ", b"\n"):
                yield b"|" * at + rare + b"|" * (m - at - 1)
    yield b"||||||| | | |||||||"
    yield b"||||\n||||\n||||"


@pytest.mark.parametrize("staged", [1, 0])
@pytest.mark.parametrize("n", [40, TILE, 2 * TILE + 301, 260 * TILE + 5])
def test_windows(parser, staged, n):
    text = np.full(n, ord("|"), np.uint8)
    rng = np.random.default_rng(n)
    edges = [e + d for e in (0, 256, TILE, 2 * TILE, 259 * TILE, n) for d in (-270, -9, -4, -1, 0, 2, 3, 8, 13, 290)]
    for i, e in enumerate([e for e in edges if 0 <= e < n] + rng.integers(0, n, 40).tolist()):
        text[e] = b"q \n"[i % 3]
    data = text.tobytes()
    doc = parser.upload(data)
    pats = [p for p in patterns() if len(p) <= n]
    was = parser.tuning["search_staged"]
    parser.set_tuning(search_staged=staged)
    try:
        for i in range(0, len(pats), 8):
            for p, r in zip(pats[i: i + 8], parser.search_document_multi(doc, pats[i: i + 8], n)):
                want = oracle.find_all(data, p)
                assert r.total_matches == len(want) and np.array_equal(r.offsets, want), (len(p), p[:70])
    finally:
        parser.set_tuning(search_staged=was)


def test_absent_rare_byte_is_cheap(parser):
    import ctypes

    import torch

    L, n = _lib.load(), 64 << 20
    stream = torch.cuda.ExternalStream(L.ol_ctx_stream(parser.ctx))
    out = torch.zeros(1024, dtype=torch.int32, device="cuda")
    total = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    doc = parser.upload(np.full(n, ord("|"), np.uint8))

    def ms(pattern):
        pat, times = ctypes.create_string_buffer(pattern, len(pattern)), []
        for _ in range(15):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            _lib.check(L.ol_search_async(parser.ctx, doc.handle, pat, len(pattern), 1024, total.data_ptr(), out.data_ptr()),
                       parser.ctx)
            b.record(stream)
            b.synchronize()
            times.append(a.elapsed_time(b))
        return float(np.median(times))

    # 1.5 times a pattern that occurs everywhere, when every place is looked at closely
    assert ms(b"||||||||a") < ms(b"||||||||")
