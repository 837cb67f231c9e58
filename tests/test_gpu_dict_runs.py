"""Dictionary search around runs of one byte (run masks, run ends, trie runs)
against the oracle: runs across slice and tile edges and the text end, several
run bytes (a line break and NUL among them), and documents of a batch that end
or begin in a run."""
import numpy as np
import pytest

import oracle
from oneline_b200 import HIT_DTYPE

pytestmark = pytest.mark.gpu

BYTES = [b"|", b"-", b" ", b"\n", b"\0", b"="]


def runs_text(seed: int, n: int) -> bytes:
    rng = np.random.default_rng(seed)
    parts, size = [], 0
    while size < n:
        c = BYTES[int(rng.integers(0, len(BYTES)))]
        k = int(rng.choice([1, 2, 3, 4, 5, 9, 33, 62, 63, 64, 65, 130, 511, 513, 1030],
                           p=[.2, .15, .15, .12, .1, .1, .04, .03, .03, .02, .02, .01, .01, .01, .01]))
        parts += [c * k, bytes(rng.integers(97, 100, int(rng.integers(0, 5)), dtype=np.uint8))]
        size += len(parts[-2]) + len(parts[-1])
    return b"".join(parts)[:n]


def patterns_of(text: bytes, seed: int, n: int) -> list:
    rng = np.random.default_rng(seed)
    pats = []
    for _ in range(n):
        m = int(rng.integers(4, 65))
        at = int(rng.integers(0, len(text) - m))
        pats.append(text[at: at + m])
    for c in BYTES:  # runs, run ends, and runs inside
        pats += [c * k for k in (4, 5, 7, 31, 32, 33, 63, 64)]
        pats += [c * r + x for r in (2, 3, 4, 5, 40, 62, 63) for x in (b"a", b"|", b" a") if c * r + x != c * (r + 1)]
        pats += [b"a" + c * r for r in (3, 4, 6, 12, 33, 63)] + [b"b\n" + c * 9, b"a\n|||" + c * 4]
    return [p for p in pats if 4 <= len(p) <= 64] + pats[:5]


def many(text: bytes, pats):
    counts, hp, ho, total = oracle.CpuBaseline(threads=8).many(pats).find_all_par(text)
    return counts.astype(np.uint64), hp, ho, int(total)


@pytest.mark.parametrize("n", [4, 511, 512, 515, 575, 16384, 16384 + 63, 70_001, 1_900_003])
@pytest.mark.parametrize("heavy_min_hits", [1, 40, 1 << 30])
def test_runs_everywhere(parser, n, heavy_min_hits):
    import torch

    text = runs_text(n, n)
    source = runs_text(n, 70_001)
    pats = patterns_of(source if n < 1000 else text, n + 1, 300)
    counts, hp, ho, total = many(text, pats)
    doc = parser.upload(text)
    ps = parser.compile_patterns(doc, pats, max_patterns=None)
    buf = torch.full((2 * max(total, 1),), -1, dtype=torch.int32, device="cuda")
    c, t = parser.search_many_device(doc, ps, buf.data_ptr(), total, heavy_min_hits=heavy_min_hits)
    hits = buf.cpu().numpy().view(HIT_DTYPE)[:total]
    assert t == total and np.array_equal(c.astype(np.uint64), counts)
    assert np.array_equal(hits["pattern"], hp) and np.array_equal(hits["offset"], ho)


@pytest.mark.parametrize("heavy_min_hits", [1, 1 << 30])
def test_runs_stay_inside_documents(parser, heavy_min_hits):
    import torch

    docs = [runs_text(s, 200 + 97 * s) for s in range(40)]
    docs += [b"|" * 700, b"", b"|" * 70 + b"\n", b"\n" * 80, b"-" * 3, b"|||a", b"\0" * 90, b"||||"]
    text = b"".join(docs)
    pats = patterns_of(text, 5, 200)
    batch = parser.upload_batch(docs)
    ps = parser.compile_patterns(None, pats)
    want_counts = np.zeros(len(pats), np.uint64)
    hits = []
    for i, d in enumerate(docs):
        if len(d) < 4:
            continue
        counts, hp, ho, _ = many(d, pats)
        want_counts += counts
        hits.append(np.stack([hp.astype(np.int64), ho.astype(np.int64) + batch.doc_info(i)[0]], 1))
    want = np.concatenate(hits)
    want = want[np.lexsort((want[:, 1], want[:, 0]))]
    buf = torch.full((len(want), 2), -1, dtype=torch.int32, device="cuda")
    c, t = parser.batch_search_many(batch, ps, buf.data_ptr(), len(want), heavy_min_hits=heavy_min_hits)
    assert t == len(want) and np.array_equal(c.astype(np.uint64), want_counts)
    assert np.array_equal(buf.cpu().numpy().astype(np.int64), want)
