"""Inputs whose k-mers are spread unevenly over the printed order, or are nearly
all distinct: sort units and rounds of every sub-bucket, sub-buckets that no
table holds, passes and batches with a few of them.  Integer work: exact
comparisons against the oracle, or plain torch where the oracle would take
minutes."""
import random

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu
U32 = 0xFFFFFFFF
BASES = np.frombuffer(b"ACGT", np.uint8)


@pytest.fixture(scope="module")
def counter():
    import ktcountermemorygreedy_b200 as kc
    with kc.KmerCounter(max_inflight_jobs=1) as c:
        yield c


def _record(seq):
    return b"@r\n" + seq + b"\n+\n" + b"I" * len(seq) + b"\n"


def _torch_records(codes, k):
    """Sorted records of one sequence of base codes (k <= 31), as k-mer words
    and counts."""
    import torch
    c = torch.from_numpy(codes).cuda().to(torch.int64)
    n = len(codes) - k + 1
    f, rc = torch.zeros(n, dtype=torch.int64, device="cuda"), torch.zeros(n, dtype=torch.int64, device="cuda")
    for i in range(k):   # first base first, and its reverse complement's word
        f = (f << 2) | c[i:i + n]
        rc |= (3 - c[i:i + n]) << (2 * i)
    # the canonical strand has the smaller last-base-first word
    def rev(x):
        r = torch.zeros_like(x)
        for i in range(k):
            r |= ((x >> (2 * i)) & 3) << (2 * (k - 1 - i))
        return r
    s = torch.where(rev(f) <= rev(rc), f, rc)
    u, cnt = torch.unique(s, return_counts=True)
    words = rev(u).cpu().numpy().astype(np.uint64) << np.uint64(64 - 2 * k)
    return words, cnt.cpu().numpy().astype(np.uint32)


@pytest.mark.parametrize("shape", [1, 2])
def test_assembly_of_distinct_kmers(counter, shape):
    """70M k-mers, nearly all distinct: sub-buckets of up to twice the table's
    slots are counted in rounds, and every round is a sort unit of its own."""
    codes = np.random.default_rng(3).integers(0, 4, 70_000_000, dtype=np.uint8)
    want_k, want_c = _torch_records(codes, 31)
    counter.set_tuning(count_shape=shape)
    r = counter.count([_record(BASES[codes].tobytes())], k=31, count_max=U32, hist_max=10)
    counter.set_tuning(count_shape=1)
    assert r.smem_passes == 1 and r.smem_fallbacks == 0
    assert np.array_equal(r.keys, want_k) and np.array_equal(r.counts, want_c)
    assert r.hist.tolist() == O.histogram(want_c, 1, 10).tolist()
