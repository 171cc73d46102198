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


def _uniform(seed, n, length=150):
    reads = BASES[np.random.default_rng(seed).integers(0, 4, size=(n, length), dtype=np.uint8)]
    return [r.tobytes() for r in reads]


def _repeat(seed, unit, n, sub, length=150):
    """Reads of a repeated unit with substitutions."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(n):
        s = np.resize(np.frombuffer(unit, np.uint8), length + len(unit))[rng.integers(0, len(unit)):][:length].copy()
        at = np.nonzero(rng.random(length) < sub)[0]
        s[at] = BASES[rng.integers(0, 4, len(at))]
        out.append(s.tobytes())
    return out


def _fastq(seqs, seed=0):
    seqs = list(seqs)
    random.Random(seed).shuffle(seqs)
    return b"".join(_record(s) for s in seqs)


def _oracle(files, k):
    return (O.exact_records if k <= 32 else O.exact_records_wide)(files, k, U32)


def _check(c, files, k, min_count=1, max_count=U32, count_max=U32, want=None, **kw):
    all_k, all_c = want or _oracle(files, k)
    cc = np.minimum(all_c, count_max)
    m = (cc >= min_count) & (cc <= max_count)
    r = c.count(files, k=k, count_max=count_max, min_count=min_count, max_count=max_count, hist_max=300_000, top_n=20, **kw)
    assert np.array_equal(r.keys, all_k[m]) and np.array_equal(r.counts, cc[m])
    assert r.hist.tolist() == O.histogram(cc, 1, 300_000).tolist()
    assert r.distinct == len(all_k) and r.occurrences == int(all_c.sum(dtype=np.uint64))
    order = np.argsort(-cc[m].astype(np.int64), kind="stable")[:20]
    assert np.array_equal(r.top_keys, all_k[m][order]) and np.array_equal(r.top_counts, cc[m][order])
    return r


@pytest.mark.parametrize("k", [16, 31, 32, 33, 63, 64, 96, 127])
def test_reads_of_repeats_are_counted_in_the_pass(counter, k):
    """Poly-A and microsatellites with errors: far more k-mers that start alike
    than a table holds, in a few of the sub-buckets.  Those are counted on their
    own, the pass stays where it is."""
    seqs = _uniform(k, 20_000, 250)
    for i, unit in enumerate((b"A", b"AC", b"GATA")):
        seqs += _repeat(100 * k + i, unit, 700, 0.03, 250)
    f = [_fastq(seqs, k)]
    want = _oracle(f, k)
    for kw in (dict(), dict(bloom=True, memory_gb=1, min_count=2), dict(count_max=3, min_count=2, max_count=3)):
        r = _check(counter, f, k, want=want, **kw)
        assert r.smem_passes == 1 and r.smem_fallbacks == 0


@pytest.mark.parametrize("k", [31, 63, 127])
@pytest.mark.parametrize("n", [262_143, 262_144, 262_145, 400_000])
def test_one_kmer_at_the_edge_of_a_blocks_share(counter, k, n):
    """n occurrences of one k-mer, at and around the number of keys that one
    block counts (262144)."""
    f = [_record(b"A" * (n + k - 1)) + _fastq(_uniform(n + k, 30_000, 250), 1)]
    r = _check(counter, f, k)
    assert r.smem_passes == 1 and r.smem_fallbacks == 0
    assert int(r.counts.max()) >= n


@pytest.mark.parametrize("shape", [1, 2])
@pytest.mark.parametrize("k", [31, 47, 101])
def test_crowded_after_finished_rounds(counter, k, shape):
    """A sub-bucket whose first rounds fit and whose last ones do not: 20000
    k-mers of one 10-base prefix spread evenly and 20000 more in its last part
    that share 26 bases."""
    rnd = random.Random(k)
    tail = lambda n: "".join(rnd.choice("ACGT") for _ in range(n))
    p = "AC" + tail(8)
    even = {p + rnd.choice("AC") + tail(k - 12) + "A" for _ in range(20_000)}
    q = p + "TT" + tail(14)
    late = {q + tail(k - 27) + "A" for _ in range(20_000)} if k > 31 else {q + tail(4) + "A" for _ in range(300)} | {
        p + "TTT" + tail(k - 14) + "A" for _ in range(20_000)}
    seqs = [s.encode() for s in even | late]
    seqs += seqs[::5] + _uniform(k, 6000, 300)
    counter.set_tuning(count_shape=shape)
    r = _check(counter, [_fastq(seqs, k)], k, min_count=1)
    counter.set_tuning(count_shape=1)
    assert r.smem_passes == 1 and r.smem_fallbacks == 0


@pytest.mark.parametrize("k", [31, 63])
def test_one_crowded_pass_of_several(counter, k):
    """A job in passes whose k-mers crowd into one prefix in one of them: only
    that pass counts most of its k-mers in global memory."""
    seqs = _uniform(5, 30_000) + _repeat(6, b"A", 6000, 0.03)
    f = [_fastq(seqs, 2)]
    r = _check(counter, f, k, pass_bytes=16 << 20)
    assert r.passes > 3 and r.smem_fallbacks == 1 and r.smem_passes == r.passes - 1


def test_crowded_samples_of_a_batch(counter):
    """Two samples with the same repeats and one without, k equal and not: each
    has its own counts, and the batch stays in shared memory."""
    seqs = [_uniform(i, 12_000) + (_repeat(9 + i // 2, b"A", 900, 0.03) if i < 3 else []) for i in range(4)]
    files = [[_fastq(s, i)] for i, s in enumerate(seqs)]
    ks = [31, 31, 25, 31]
    rs = counter.count_batch(files, ks, count_max=U32, hist_max=200_000)
    for f, k, r in zip(files, ks, rs):
        all_k, all_c = _oracle(f, k)
        assert np.array_equal(r.keys, all_k) and np.array_equal(r.counts, all_c)
        assert r.hist.tolist() == O.histogram(all_c, 1, 200_000).tolist()
        assert r.distinct == len(all_k) and r.smem_passes == 1 and r.smem_fallbacks == 0


@pytest.mark.parametrize("k", [63, 96, 127])
@pytest.mark.parametrize("large", [False, True])
def test_sampled_regions_of_long_kmers_fit(counter, k, large):
    """Sub-buckets of two- and four-word k-mers are small, and regions estimated
    from a sample leave each a margin that the key arrays have no room for, with
    an exact census or (from 4 MiB on) a sampled one: such passes count exactly
    instead of scattering twice."""
    f = [_fastq(_uniform(k, 27_000 if large else 8_000, 250))]
    assert (len(f[0]) > 4 << 20) == large
    counter.set_tuning(sampled_region_keys=1)
    r = _check(counter, f, k)
    counter.set_tuning(sampled_region_keys=64 << 20)
    assert r.smem_passes == 1 and r.region_redos == 0


def _tiles(seqs):
    """One record per 8 KiB tile of the input."""
    out = []
    for s in seqs:
        out.append(b"@rr\n" + s + b"\n+\n" + b"I" * 4092 + b"\n")
        assert len(out[-1]) == 8192
    return b"".join(out)


@pytest.mark.parametrize("k", [31, 63, 127])
@pytest.mark.parametrize("resident", [False, True])
def test_census_sample_unlike_the_rest(counter, k, resident):
    """Every eighth tile, those of the census sample, is unlike the others: the
    buckets outgrow their regions, and the input that is on the device already
    is counted again."""
    rng = np.random.default_rng(k)
    f = _tiles(BASES[rng.integers(0, 4, 4092)].tobytes() if i % 8 == 0 else np.resize(BASES[rng.integers(0, 4, 97)], 4092).tobytes()
               for i in range(600))
    want_k, want_c = _oracle([f], k)
    kw = dict(k=k, count_max=U32, hist_max=10)
    if resident:
        inp = counter.upload([f])
        r = counter.count(input=inp, **kw)
        counter.free_input(inp)
    else:
        r = counter.count([f], **kw)
    assert np.array_equal(r.keys, want_k) and np.array_equal(r.counts, want_c)
    assert r.hist.tolist() == O.histogram(want_c, 1, 10).tolist()


def test_streamed_upload_whose_first_quarter_is_unlike_the_rest(counter):
    """A file that goes up in chunks: its first quarter, from which the bucket
    regions come, has A and T only."""
    rng = np.random.default_rng(8)
    codes = rng.integers(0, 4, 280_000_000, dtype=np.uint8)
    codes[: 70_000_000] = 3 * (codes[: 70_000_000] & 1)
    f = _record(BASES[codes].tobytes())
    assert len(f) > 512 << 20
    want_k, want_c = _torch_records(codes, 31)
    for kw in (dict(), dict(bloom=True, memory_gb=8)):
        r = counter.count([f], k=31, count_max=U32, hist_max=10, **kw)
        assert r.occurrences == len(codes) - 30
        assert np.array_equal(r.keys, want_k) and np.array_equal(r.counts, want_c)


@pytest.mark.parametrize("k,length", [(31, 34), (63, 66), (127, 130)])
def test_few_kmers_in_many_tiles(counter, k, length):
    """Reads hardly longer than k: the census sample of 600 tiles holds few
    k-mers."""
    n = 600 * 8192 // (2 * length + 7)
    f = _fastq(_uniform(k, n // 2, length) + _uniform(k + 1, n - n // 2 + 100, min(length, k - 2)), 3)
    r = _check(counter, [f], k)
    assert r.smem_passes == 1 and r.smem_fallbacks == 0


_LITTLE_MEMORY = """
import sys
import numpy as np, torch
import ktcountermemorygreedy_b200 as kc
k, n = int(sys.argv[1]), int(sys.argv[2])
free, _ = torch.cuda.mem_get_info()
held = torch.empty(free - (5 << 30), dtype=torch.uint8, device="cuda")
with kc.KmerCounter(max_inflight_jobs=1) as c:
    f = b"@r\\n" + b"A" * n + b"\\n+\\n" + b"I" * n + b"\\n"
    r = c.count([f], k=k, count_max=kc.U32_MAX)
    assert r.occurrences == n - k + 1 and r.distinct == 1, (r.occurrences, r.distinct)
    assert r.counts.tolist() == [n - k + 1] and not r.keys.any()
    assert r.smem_passes == 0 and r.smem_fallbacks == 1
"""


@pytest.mark.parametrize("k,n", [(31, 260_000_000), (63, 140_000_000)])
def test_occurrences_that_do_not_fit_the_device(k, n):
    """One k-mer's occurrences larger than the device memory left (5 GB, the
    rest is held), its table a few slots: counted in global-memory tables."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", _LITTLE_MEMORY, str(k), str(n)], cwd=root, capture_output=True, text=True,
                       timeout=300)
    assert p.returncode == 0, p.stderr[-2000:]


@pytest.mark.parametrize("k,n,shared", [(31, 7000, 24), (31, 7000, 16), (63, 3500, 42), (127, 1700, 42)])
def test_sort_unit_of_one_run(counter, k, n, shared):
    """A unit whose records all share the sort's digit but one: each is ranked
    among all others.  24 shared bases of 31 leave 4096 k-mers that follow one
    another, which crowd the table's slots too and may be counted apart."""
    rnd = random.Random(k)
    tail = lambda m: "".join(rnd.choice("ACGT") for _ in range(m))
    p = "AC" + tail(shared - 2)
    if shared == 24:
        seqs = [p + "".join("ACGT"[(i >> 2 * j) & 3] for j in range(6)) + "A" for i in range(4096)]
    else:
        seqs = list({p + tail(k - shared - 1) + "A" for _ in range(n)})
    seqs.append(p[:6] + ("T" if p[6] != "T" else "G") + tail(k - 8) + "A")
    seqs += seqs[:100]
    r = _check(counter, [_fastq([s.encode() for s in seqs])], k)
    if shared != 24:
        assert r.smem_passes == 1 and r.smem_fallbacks == 0


def test_more_small_units_than_their_list(counter):
    """128 sub-buckets that need all 64 rounds, 62 of them with a single k-mer:
    more units of the smallest size than their list holds at first."""
    rng = np.random.default_rng(6)
    keys = []
    for b in range(64):                       # buckets A...: with a last base A the forward strand is canonical
        for sub in (1, 3):                    # of 4
            r = np.concatenate([np.repeat(np.uint64([10, 11]), 5000), np.uint64([x for x in range(64) if x not in (10, 11)])])
            t = rng.integers(0, 1 << 44, len(r), dtype=np.uint64) << np.uint64(2)
            keys.append((np.uint64(b) << np.uint64(54)) | (np.uint64(sub) << np.uint64(52)) | (r << np.uint64(46)) | t)
    keys = rng.permutation(np.unique(np.concatenate(keys)))
    codes = (keys[:, None] >> np.arange(60, -2, -2, dtype=np.uint64)) & np.uint64(3)
    seq = np.full((len(keys), 69), 10, np.uint8)   # @ r \n, 31 bases, \n + \n, 31 qualities, \n
    seq[:, :3] = np.frombuffer(b"@r\n", np.uint8)
    seq[:, 3:34] = BASES[codes]
    seq[:, 34:37] = np.frombuffer(b"\n+\n", np.uint8)
    seq[:, 37:68] = 73
    r = _check(counter, [seq.tobytes()], 31)
    assert len(r.counts) == len(keys) and r.smem_passes == 1 and r.smem_fallbacks == 0


def test_large_sub_buckets_of_a_large_pass(counter):
    """150M k-mers, so that one block may count up to 586K keys, in one round
    from 262144 on: two frequent k-mers (counted in it), a repeat with errors
    (too many distinct ones for it) and a run beyond the limit."""
    rng = np.random.default_rng(12)
    codes = rng.integers(0, 4, 150_000_000, dtype=np.uint8)
    codes[10_000_000:10_400_000] = 2                                   # G
    codes[20_000_000:20_900_000] = np.resize(np.uint8([0, 1]), 900_000)   # AC and CA, 450K each
    codes[30_000_000:31_000_000] = 0                                   # A, beyond the limit
    errors = np.resize(np.uint8([0, 3]), 1_000_000)                    # AT with errors
    at = rng.integers(0, len(errors), 30_000)
    errors[at] = rng.integers(0, 4, len(at))
    codes[40_000_000:41_000_000] = errors
    want_k, want_c = _torch_records(codes, 31)
    r = counter.count([_record(BASES[codes].tobytes())], k=31, count_max=U32, hist_max=2_000_000)
    assert r.smem_passes == 1 and r.smem_fallbacks == 0
    assert np.array_equal(r.keys, want_k) and np.array_equal(r.counts, want_c)
    assert r.hist.tolist() == O.histogram(want_c, 1, 2_000_000).tolist()


def test_crowded_jobs_side_by_side():
    """Jobs with crowded sub-buckets on several workers of one handle: each has
    the results it has alone."""
    import ktcountermemorygreedy_b200 as kc
    jobs = [(k, [_fastq(_uniform(i, 9000) + _repeat(50 + i, (b"A", b"AC", b"GATA")[i % 3], 800, 0.03), i)])
            for i, k in enumerate((31, 63, 25, 127, 31, 47, 32, 31))]
    with kc.KmerCounter(max_inflight_jobs=1) as c:
        alone = [c.count(f, k=k, count_max=U32, hist_max=100) for k, f in jobs]
    with kc.KmerCounter(max_inflight_jobs=4) as c:
        ids = [c.submit(f, k=k, count_max=U32, hist_max=100) for _ in range(3) for k, f in jobs]
        for i, (j, (k, _)) in enumerate(zip(ids, jobs * 3)):
            c.wait(j)
            r, want = c.result(j, k), alone[i % len(jobs)]
            assert np.array_equal(r.keys, want.keys) and np.array_equal(r.counts, want.counts)
            assert np.array_equal(r.hist, want.hist)
