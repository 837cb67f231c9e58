"""A dictionary search on a GPU that is nearly full: where the bitmaps of all the
patterns that might be frequent do not fit, it makes do with those of the patterns
that are."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# In a process of its own, with a memory pool that holds nothing else. 32 bitmaps
# of 60 MiB of text are 240 MiB; one (there is one frequent pattern) is 7.5.
SEARCH = """
import numpy as np, torch
from oneline_b200 import GpuParser

MIB = 1 << 20
n, leave = 60 * MIB, 144 * MIB
text = np.random.default_rng(3).integers(97, 123, n, dtype=np.uint8)
text[4096: 4096 + MIB] = ord("|")
at = [100, 2 * MIB, 9 * MIB + 5, n - 12]
pats = [b"||||"] + [text[a: a + 12].tobytes() for a in at] + [b"zzzz-absent-%d" % i for i in range(40)]
want = [MIB - 3] + [1] * len(at) + [0] * 40
parser = GpuParser(0)
patterns = parser.compile_patterns(None, pats)
small = parser.upload(text[: 2 * MIB].tobytes())
parser.search_many(small, patterns, 64)  # the kernels are loaded
doc = parser.upload(text.tobytes())
held, part = [], torch.cuda.mem_get_info()[0] - leave
while part > 2 * MIB and torch.cuda.mem_get_info()[0] > leave + 8 * MIB:
    try:
        held.append(torch.empty(min(part, torch.cuda.mem_get_info()[0] - leave), dtype=torch.uint8, device="cuda"))
    except torch.OutOfMemoryError:
        part //= 2
assert torch.cuda.mem_get_info()[0] < 200 * MIB
for _ in range(2):
    r = parser.search_many(doc, patterns, 1 << 16)
    assert r.counts.tolist() == want and r.total_hits == sum(want)
    assert np.array_equal(r.hits["offset"], np.arange(1 << 16) + 4096) and not r.hits["pattern"].any()
print("searched with", torch.cuda.mem_get_info()[0] // MIB, "MiB free")
"""


def test_search_with_little_memory_left():
    r = subprocess.run([sys.executable, "-c", SEARCH], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "searched with" in r.stdout, r.stdout + r.stderr[-3000:]
