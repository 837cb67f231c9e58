"""The page-locked buffer that short results come back through: it grows seldom,
to at most twice what was asked for, and answers that get larger and smaller from
call to call on one parser are whole, around the sizes (64 KiB, 1 MiB) at which
the way back changes."""
import ctypes

import numpy as np
import pytest

from oneline_b200 import GpuParser, _lib

pytestmark = pytest.mark.gpu


class HostBuf(ctypes.Structure):  # ol::HostBuf
    _fields_ = [("ptr", ctypes.c_void_p), ("bytes", ctypes.c_size_t)]


def test_growing_needs_seldom_allocate(parser):
    L = _lib.load()
    reserve, release = L["_ZN2ol7HostBuf7reserveEm"], L["_ZN2ol7HostBuf7releaseEv"]
    reserve.argtypes, release.argtypes = [ctypes.c_void_p, ctypes.c_size_t], [ctypes.c_void_p]
    release.restype = None
    buf, sizes = HostBuf(), set()
    for need in range(4, (1 << 20) + 1, 4092):
        assert reserve(ctypes.byref(buf), need) == 0 and buf.bytes >= need
        sizes.add(buf.bytes)
    assert len(sizes) <= 6 and buf.bytes <= 2 << 20, sizes
    release(ctypes.byref(buf))
    assert not buf.ptr and buf.bytes == 0


def test_answers_of_changing_size():
    n = 300_000
    text = np.tile(np.frombuffer(b"a\n|b", np.uint8), n)
    at = {b"a": np.arange(n, dtype=np.uint32) * 4, b"|": np.arange(n, dtype=np.uint32) * 4 + 2}
    parser = GpuParser(0)
    doc = parser.upload(text)
    around = [m + d for m in (1 << 14, 1 << 18) for d in (-65, -1, 0, 1)]
    for room in [1, 100, *around, 262_144 // 2, 300_001, 5, *around[::-1]]:
        r = parser.search_document(doc, b"a", room)
        assert r.total_matches == n and np.array_equal(r.offsets, at[b"a"][:room])
        for p, r in zip((b"|", b"zz", b"a"), parser.search_document_multi(doc, [b"|", b"zz", b"a"], room)):
            assert np.array_equal(r.offsets, at.get(p, np.zeros(0, np.uint32))[:room])
        q = parser.query_document(doc, 1, 0, room)  # the first line: "a"; all others are "|ba"
        assert q.total_matches == 1 and q.indices.tolist() == [0]
        q = parser.query_document(doc, 1, 1, room)
        assert q.total_matches == n and np.array_equal(q.indices, np.arange(1, n + 1)[:room])
    parser.close()
