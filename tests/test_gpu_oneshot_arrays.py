"""The result arrays of a one-shot parse keep room for at most twice the lines (or
4096), whatever was guessed for them, and a host that does not give that much is asked for
the exact size."""
import numpy as np
import pytest

import oracle
from oneline_b200 import gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 40, 5000, 300_000, (1 << 21) + 7])
@pytest.mark.parametrize("line", [b"\n", b"|a\n", b"| an entry of some length, as most lines are\n"])
def test_arrays_are_not_much_larger_than_the_lines(parser, monkeypatch, n, line):
    text = np.resize(np.frombuffer(line, np.uint8), n).tobytes()
    offs, nodes = oracle.parse(text)

    def check():
        tree, scan = parser.parse_raw(text), parser.scan_line_offsets(text)
        for got, want in ((tree.line_offsets, offs), (tree.nodes, nodes), (scan, offs)):
            assert np.array_equal(got, want) and got.dtype == want.dtype
            whole = got if got.base is None else got.base
            assert whole.size <= max(2 * want.size + 1, 4096)

    check()
    empty = np.empty

    def scarce(shape, *args, **kwargs):
        if shape > len(offs):
            raise MemoryError
        return empty(shape, *args, **kwargs)

    monkeypatch.setattr(gpu.np, "empty", scarce)
    check()
