"""Tree links around the sizes at which the tiles and passes change: one tile,
tiles of 1024 lines up to 64 of them, tiles of 4096 lines with and without the
scan pass, against the oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def lines_text(n: int, levels: int) -> bytes:
    rng = np.random.default_rng(n * 31 + levels)
    depth = np.abs(np.cumsum(rng.integers(-2, 3, n))) % levels
    depth[rng.integers(0, n, max(n // 5000, 1))] = 0  # a few far-away ancestors
    blank = rng.random(n) < 0.15
    return b"".join(b"|" * int(d) + (b"\n" if e else b" x\n") for d, e in zip(depth, blank))


@pytest.mark.parametrize("levels", [1, 2, 17, 32])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 1024, 1025, 2049, 64 * 1024 - 1, 64 * 1024, 64 * 1024 + 1, 64 * 1024 + 9,
                               64 * 4096 - 3, 64 * 4096, 64 * 4096 + 1])
def test_sizes(parser, n, levels):
    text = lines_text(n, levels)
    _, nodes = oracle.parse(text)
    assert len(nodes) == n
    got = parser.download_tree(parser.build_tree(parser.upload(text)))
    want = oracle.full_tree(nodes)
    for k in want:
        assert np.array_equal(got[k], want[k]), k


def deep_text(n: int, shape: str) -> bytes:
    rng = np.random.default_rng(n)
    if shape == "walk":
        depth = np.abs(np.cumsum(rng.integers(-3, 4, n)) % 120 - 60) + 3
    elif shape == "random":
        depth = rng.integers(0, 300 if n < 5000 else 45, n)
    elif shape == "flat":  # every search goes to the ends of the document
        depth = np.full(n, 40)
    else:  # sawtooth: parents and ends far away
        depth = 50 - np.arange(n) * 50 // n + (np.arange(n) % 3 == 0)
    depth[n // 2] = 33
    blank = rng.random(n) < 0.2
    return b"".join((b"|" * int(d) + (b"\n" if e else b" x\n")) if d or not e else b"\n" for d, e in zip(depth, blank))


@pytest.mark.parametrize("shape", ["walk", "random", "flat", "sawtooth"])
@pytest.mark.parametrize("n", [2, 31, 33, 1023, 1024, 1025, 3000, 32 * 1024 - 1, 32 * 1024 + 1, 200_001])
def test_any_depth(parser, n, shape):
    text = deep_text(n, shape)
    _, nodes = oracle.parse(text)
    assert len(nodes) == n
    got = parser.download_tree(parser.build_tree(parser.upload(text), strict_depth=False))
    want = oracle.full_tree(nodes)
    for k in want:
        assert np.array_equal(got[k], want[k]), k
