"""Patterns that are one byte repeated, of rare and common bytes and of every
length up to the longest that is staged and past it, in texts of runs around that
length, across tile edges and up to the text's end; and what they cost."""
import numpy as np
import pytest

from oneline_b200 import _lib

pytestmark = pytest.mark.gpu

TILE = 16384
LENGTHS = [8, 15, 16, 47, 48, 49, 50, 62, 63, 64, 65, 79, 80, 96, 200, 1000, 4081, 4095, 4096, 4097]


def runs_of(mask: np.ndarray, m: int) -> np.ndarray:
    edge = np.diff(np.concatenate([[0], mask.view(np.int8), [0]]))
    parts = [np.arange(s, e - m + 1) for s, e in zip(np.nonzero(edge == 1)[0], np.nonzero(edge == -1)[0]) if e - s >= m]
    return np.concatenate(parts).astype(np.uint32) if parts else np.zeros(0, np.uint32)


def text_of(byte: int, tiles: int, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    parts, size = [], 0
    while size < tiles * TILE:
        m = int(rng.choice(LENGTHS)) + int(rng.integers(-1, 3)) + (16 * int(rng.integers(0, 3)) if rng.random() < 0.3 else 0)
        parts += [np.full(m, byte, np.uint8), rng.integers(97, 123, int(rng.integers(1, 20)), dtype=np.uint8)]
        size += parts[-2].size + parts[-1].size
    text = np.concatenate(parts)[: tiles * TILE]
    text[3 * TILE - 5000: 3 * TILE + 7000] = byte
    text[-5003:] = byte  # up to the end, past which the buffer is zero
    return text


@pytest.mark.parametrize("byte", [ord("|"), ord("Z"), 0])
@pytest.mark.parametrize("staged", [1, 0])
@pytest.mark.parametrize("tiles,cut", [(5, 0), (5, 4001), (260, 77)])
def test_runs(parser, byte, staged, tiles, cut):
    text = text_of(byte, tiles, tiles + byte)[: tiles * TILE - cut]
    doc = parser.upload(text)
    mask = text == byte
    was = parser.tuning["search_staged"]
    parser.set_tuning(search_staged=staged)
    try:
        for i in range(0, len(LENGTHS), 7):
            some = LENGTHS[i: i + 7]
            got = parser.search_document_multi(doc, [bytes([byte]) * m for m in some], text.size)
            for m, r in zip(some, got):
                want = runs_of(mask, m)
                assert r.total_matches == want.size and np.array_equal(r.offsets, want), m
    finally:
        parser.set_tuning(search_staged=was)


def test_cost_does_not_depend_on_the_byte_or_grow_with_the_length(parser):
    import ctypes

    import torch

    L, n = _lib.load(), 64 << 20
    stream = torch.cuda.ExternalStream(L.ol_ctx_stream(parser.ctx))
    out = torch.zeros(1024, dtype=torch.int32, device="cuda")
    total = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()

    def ms(byte, m):
        doc, pat = parser.upload(np.full(n, byte, np.uint8)), ctypes.create_string_buffer(bytes([byte]) * m, m)
        times = []
        for _ in range(15):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            _lib.check(L.ol_search_async(parser.ctx, doc.handle, pat, m, 1024, total.data_ptr(), out.data_ptr()), parser.ctx)
            b.record(stream)
            b.synchronize()
            times.append(a.elapsed_time(b))
        assert int(total.item()) == n - m + 1
        return float(np.median(times))

    short = ms(ord("|"), 8)
    assert ms(ord("Z"), 8) < 2 * short  # 5 times by anchor words
    assert ms(ord("|"), 64) < 4 * short  # 19 times start by start
