"""Patterns of 5 to 7 bytes, looked for by their first two: beginnings that are
everywhere, occurrences across pieces and tiles and at the text's end (past which
the buffer is zero), against the oracle; and what absent ones cost."""
import numpy as np
import pytest

import oracle
from oneline_b200 import _lib

pytestmark = pytest.mark.gpu

TILE = 16384


@pytest.mark.parametrize("staged", [1, 0])
@pytest.mark.parametrize("n", [7, 33, TILE, 2 * TILE + 6, 260 * TILE + 3])
def test_mids(parser, staged, n):
    rng = np.random.default_rng(n)
    text = rng.choice(np.frombuffer(b"ab\0", np.uint8), n)
    at = rng.integers(0, n, n // 9)
    text[at] = ord("a")
    for e in (16, TILE, 2 * TILE, 259 * TILE):  # a run and an alternation across the edge
        if e + 40 < n:
            text[e - 30: e - 4], text[e - 4: e + 40] = ord("a"), np.resize(np.frombuffer(b"ab", np.uint8), 44)
    text[max(0, n - 9):] = 0
    data = text.tobytes()
    pats = [b"aaaaa", b"aaaaaa", b"aaaaaaa", b"ababa", b"bababab", b"aabab", b"\0\0\0\0\0", b"\0\0\0\0\0\0\0", b"a\0\0\0\0", b"ab\0aa"]
    pats += [data[-5:], data[-6:], data[-7:], data[:7], data[: n // 2][-6:], b"zzzzzz"]
    pats = [p for p in pats if 5 <= len(p) <= n]
    doc = parser.upload(data)
    was = parser.tuning["search_staged"]
    parser.set_tuning(search_staged=staged)
    try:
        for i in range(0, len(pats), 8):
            for p, r in zip(pats[i: i + 8], parser.search_document_multi(doc, pats[i: i + 8], n)):
                want = oracle.find_all(data, p)
                assert r.total_matches == len(want) and np.array_equal(r.offsets, want), p
        for p in pats[:3]:  # alone
            r = parser.search_document(doc, p, n)
            assert np.array_equal(r.offsets, oracle.find_all(data, p)), p
    finally:
        parser.set_tuning(search_staged=was)


def test_absent_ones_are_cheaper_than_shorter(parser):
    import ctypes

    import torch

    L, n = _lib.load(), 64 << 20
    stream = torch.cuda.ExternalStream(L.ol_ctx_stream(parser.ctx))
    doc = parser.upload(np.random.default_rng(1).integers(48, 58, n, dtype=np.uint8))
    outs = [torch.zeros(64, dtype=torch.int32, device="cuda") for _ in range(8)]
    totals = torch.zeros(8, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()

    def ms(m):
        bufs = [ctypes.create_string_buffer(bytes([65 + i]) * 2 + b"xyzwv"[: m - 2], m) for i in range(8)]
        P = (ctypes.c_void_p * 8)(*[ctypes.addressof(b) for b in bufs])
        O = (ctypes.c_void_p * 8)(*[o.data_ptr() for o in outs])
        lens, rooms, times = np.full(8, m, np.uint32), np.full(8, 64, np.uint32), []
        for _ in range(15):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            _lib.check(L.ol_search_multi_async(parser.ctx, doc.handle, P, lens.ctypes.data, 8, rooms.ctypes.data,
                                               totals.data_ptr(), O), parser.ctx)
            b.record(stream)
            b.synchronize()
            times.append(a.elapsed_time(b))
        return float(np.median(times))

    assert ms(6) < 0.9 * ms(4)  # the same when four bytes are compared at every start
