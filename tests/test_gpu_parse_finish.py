"""The passes that write the line arrays: texts of at most 1024 tiles of 16 KiB
are finished in one launch, larger ones in three; lines that run past a tile's
halo, tiles with more lines than a slot holds, and line arrays that turn out too
small, against the oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

TILE = 16384
LIMIT = 1024 * TILE


def text_of(kind: str, n: int) -> bytes:
    if kind == "one line":
        return (b"|| | - " + b"x" * n)[: n - 1] + b"\r"
    if kind == "dense":  # more than 1024 lines a tile, and more lines than a first guess allows for
        return (b"|a\n" * (n // 3 + 1))[:n]
    if kind == "long":  # lines over several tiles
        return ((b"||| -. " + b"y" * 40000 + b"\r\r\n") * (n // 40000 + 1))[:n]
    # long lines that end in a dense tile, some of them starting in one
    part = b"|@" + b"z" * (2 * TILE + 37) + b"\n" + b"\n|\n" * 4000 + b"| =" + b"w" * 300
    return (part * (n // len(part) + 1))[:n]


@pytest.mark.parametrize("kind", ["one line", "dense", "long", "mixed"])
@pytest.mark.parametrize("n", [5, TILE, TILE + 256, TILE + 257, 3 * TILE + 1, LIMIT - 1, LIMIT, LIMIT + 1])
def test_line_arrays(parser, kind, n):
    import torch

    text = text_of(kind, n)
    assert len(text) == n
    offs, nodes = oracle.parse(text)
    dev = torch.from_numpy(np.frombuffer(text, np.uint8).copy()).cuda()
    torch.cuda.synchronize()
    content = nodes["depth"][nodes["kind"] != 0]
    for doc in (parser.upload_device(dev.data_ptr(), n), parser.upload(text)):
        assert np.array_equal(doc.read_offsets(), offs)
        assert np.array_equal(doc.read_kinds(), nodes["kind"].astype(np.uint8))
        assert doc.max_depth() == (int(content.max()) if content.size else 0)
        got = parser.download_tree(parser.build_tree(doc))
        want = oracle.full_tree(nodes)
        for k in want:
            assert np.array_equal(got[k], want[k]), k
