"""Batches from page-locked memory are laid out on the device: every byte of
documents of awkward sizes, at every relative alignment, against the oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("skip", [0, 1, 5, 18])
def test_every_alignment(parser, skip):
    import torch

    rng = np.random.default_rng(skip)
    sizes = [0, 1, 2, 15, 16, 17, 31, 33, 100, 0, 4095, 65535, 65536, 65537, 131072 + 7, 3] + rng.integers(1, 300, 200).tolist()
    offs = np.zeros(len(sizes) + 1, np.uint64)
    offs[1:] = np.cumsum(sizes)
    offs += np.uint64(skip)
    data = torch.empty(int(offs[-1]), dtype=torch.uint8, pin_memory=True).numpy()
    data[:] = rng.integers(97, 123, data.size)
    data[rng.integers(0, data.size, data.size // 40)] = 10
    docs = [data[int(a): int(b)].tobytes() for a, b in zip(offs[:-1], offs[1:])]
    batch = parser.upload_batch((data, offs))
    for i, d in enumerate(docs):
        got = parser.read_batch_doc(batch, i, tree=False)
        want, nodes = oracle.parse(d)
        assert np.array_equal(got["offsets"], want) and np.array_equal(got["kinds"], nodes["kind"].astype(np.uint8)), i
    # every 64-byte stretch of the larger documents occurs where it was
    pats, at = [], []
    for i, d in enumerate(docs):
        for p in range(0, len(d) - 64 if len(d) > 4000 else 0, 61):
            pats.append(d[p: p + 64])
            at.append(batch.doc_info(i)[0] + p)
    ps = parser.compile_patterns(None, pats, max_patterns=None)
    buf = torch.full((len(pats), 2), -1, dtype=torch.int32, device="cuda")
    counts, total = parser.batch_search_many(batch, ps, buf.data_ptr(), len(pats))
    assert total == len(pats) and np.all(counts == 1)
    assert np.array_equal(buf.cpu().numpy()[:, 1], np.array(at))
