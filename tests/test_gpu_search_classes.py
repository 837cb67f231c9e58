"""Substring search by every way a pattern is found (whole, by anchor words, by
its rarest four bytes, as a run of one byte), at tile edges, in texts finished in
one launch and in four, staged and recomputing, against the oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

TILE = 16384


def text_of(n: int) -> bytes:
    rng = np.random.default_rng(n)
    parts, size = [], 0
    while size < n:
        c = [b"|", b" ", b"-", b"\0", b"\n"][int(rng.integers(0, 5))]
        k = int(rng.choice([1, 2, 3, 7, 8, 9, 16, 47, 48, 49, 50, 300], p=[.2, .15, .15, .1, .1, .1, .1, .03, .02, .02, .02, .01]))
        parts += [c * k, bytes(rng.integers(97, 101, int(rng.integers(0, 30)), dtype=np.uint8))]
        size += len(parts[-2]) + len(parts[-1])
    text = bytearray(b"".join(parts)[:n])
    far = b"|" * 500 + b"QZXW" + b"|" * 20  # its rare bytes lie past the reach of anchors and windows
    for at in range(TILE - 600, n - len(far), 5 * TILE + 211):
        text[at: at + len(far)] = far
    return bytes(text)


def patterns_of(text: bytes) -> list:
    pats = [c * m for c in (b"|", b" ", b"\0") for m in (1, 4, 5, 6, 7, 8, 9, 15, 16, 17, 47, 48, 49, 64, 300)]
    pats += [b"|||||||a", b"a|||||||", b"|||||||| ", b"        |", b"||||a||||", b"| | | | | ", b"||||||||||||||||||||b", b"--------c",
             b"\0\0\0\0\0\0\0\0a", b"|" * 500 + b"QZXW", b"|" * 260 + b"QZXW||", b"QZXW" + b"|" * 20, b"|" * 4096, b"|" * 4200]
    rng = np.random.default_rng(7)
    for m in (2, 3, 5, 6, 7, 8, 9, 11, 12, 13, 31, 64, 65, 250, 1000):
        for back in (0, 1, m // 2, m - 1):
            at = TILE - back
            if at + m <= len(text):
                pats.append(text[at: at + m])
        if len(text) > m:
            at = int(rng.integers(0, len(text) - m))
            pats.append(text[at: at + m])
            pats.append(text[-m:])
    return [p for p in pats if len(p) <= len(text)]


@pytest.mark.parametrize("staged", [1, 0])
@pytest.mark.parametrize("n", [700, TILE, TILE + 1, 3 * TILE - 5, 256 * TILE - 3, 257 * TILE + 9])
def test_every_class(parser, n, staged):
    text = text_of(n)
    pats = patterns_of(text)
    doc = parser.upload(text)
    keep = parser.tuning
    parser.set_tuning(search_staged=staged)
    try:
        room = max(n // 2, 8)
        for i in range(0, len(pats), 8):
            got = parser.search_document_multi(doc, pats[i: i + 8], room)
            for p, r in zip(pats[i: i + 8], got):
                want = oracle.find_all(text, p)
                assert r.total_matches == want.size, (p[:70], len(p))
                assert np.array_equal(r.offsets, want[:room]), (p[:70], len(p))
    finally:
        parser.set_tuning(**keep)
