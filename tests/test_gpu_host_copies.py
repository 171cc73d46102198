"""Calls on a caller's arrays, around the size from which pageable memory is
copied through pinned chunks (4 MiB, chunks of 1 MiB): sizes at and beside the
edges, arrays off the page grid, pinned memory, several threads at once.
Integer work: exact comparisons."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIN = (4 << 20) // 8   # keys from which the key array is copied in chunks


def _records(n, seed):
    rng = np.random.default_rng(seed)
    return rng.permutation(n).astype(np.uint64) * 977 + 5, rng.integers(1, 2000, n).astype(np.uint32)


@pytest.mark.parametrize("n", [MIN - 1, MIN, MIN + 1, MIN + (1 << 17), 2 * MIN - 1, 2 * MIN + 3, 3_000_001])
def test_sorted_records_at_chunk_edges(n):
    import ktcountermemorygreedy_b200 as kc
    keys, counts = _records(n, n)
    order = np.argsort(keys)
    for f in (kc.sort_records, kc.sort_distinct_records):
        k, c = f(keys, counts, 40)
        assert np.array_equal(k, keys[order]) and np.array_equal(c, counts[order])


@pytest.mark.parametrize("n", [0, 1, 3, 130_000, 140_000, 700_001])
def test_dump_and_merge(n):
    import ktcountermemorygreedy_b200 as kc
    k = 29
    keys, counts = _records(n, n + 1)
    text = kc.dump_bytes(keys, counts, k)
    assert type(text) is bytes
    lines = text.split(b"\n")
    assert lines.pop() == b"" and len(lines) == n
    for i in set(range(0, n, 997)) | ({n - 1} if n else set()):
        w = int(keys[i])
        s = "".join("ACGT"[(w >> (64 - 2 * k + 2 * b)) & 3] for b in range(k))
        assert lines[i] == f"{s}\t{counts[i]}".encode()
    assert len(text) == int((k + 2 + np.floor(np.log10(np.maximum(counts, 1))).astype(np.int64) + 1).sum())
    # a merge without low k-mers, and one without high ones, of off-grid arrays
    top = np.empty(n + 1, np.uint64)[1:]
    top[:] = keys << np.uint64(64 - 2 * k)
    mk, mc, _ = kc.merge_records(top, counts, np.zeros(0, np.uint64), k, 5000)
    assert sorted(zip(mk.tolist(), mc.tolist())) == sorted(zip(top.tolist(), counts.tolist()))
    mk, mc, h = kc.merge_records(np.zeros(0, np.uint64), np.zeros(0, np.uint32), top, k, 5000)
    assert sorted(mk.tolist()) == sorted(top.tolist()) and (mc == 1).all() and h[0] == n


def test_pinned_arrays_and_threads():
    import torch

    import ktcountermemorygreedy_b200 as kc
    n = 2 * MIN + 77
    jobs = [_records(n, s) for s in range(6)]
    want = [(k[np.argsort(k)], c[np.argsort(k)]) for k, c in jobs]
    with ThreadPoolExecutor(6) as ex:
        got = list(ex.map(lambda j: kc.sort_records(j[0], j[1], 40), jobs))
    assert all(np.array_equal(g[0], w[0]) and np.array_equal(g[1], w[1]) for g, w in zip(got, want))
    hk = torch.from_numpy(jobs[0][0].view(np.int64)).pin_memory()
    hc = torch.from_numpy(jobs[0][1].view(np.int32)).pin_memory()
    text = kc.dump_bytes(hk.numpy().view(np.uint64), hc.numpy().view(np.uint32), 31)
    assert text == kc.dump_bytes(jobs[0][0], jobs[0][1], 31)
