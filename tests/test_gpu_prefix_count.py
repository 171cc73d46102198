"""Counting by printed-order prefix in shared memory, where it can go wrong: k below and at the
bucket prefix, k-mers that share a long prefix (tables counted in rounds,
buckets cut again, the global-memory fallback), one k-mer of very many
occurrences, and sort units of every size class.  Integer work: exact
comparisons against the oracle."""
import random

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu
U32 = 0xFFFFFFFF


@pytest.fixture(scope="module")
def counter():
    import ktcountermemorygreedy_b200 as kc
    with kc.KmerCounter(max_inflight_jobs=1) as c:
        yield c


def _fastq(seqs):
    return "".join(f"@r{i}\n{s}\n+\n{'I' * len(s)}\n" for i, s in enumerate(seqs)).encode()


def _check(c, fq, k, min_count=1, **kw):
    all_k, all_c = O.exact_records([fq], k, U32)
    m = all_c >= min_count
    r = c.count([fq], k=k, count_max=U32, min_count=min_count, hist_max=300, top_n=20, want_le2=True, **kw)
    assert np.array_equal(r.keys, all_k[m]) and np.array_equal(r.counts, all_c[m])
    assert r.hist.tolist() == O.histogram(all_c, 1, 300).tolist()
    assert r.distinct == len(all_k) and r.occurrences == int(all_c.sum(dtype=np.uint64))
    le = all_c[m] <= 2
    assert np.array_equal(r.le2_keys, all_k[m][le])
    if kw.get("bloom"):
        assert r.low_len + r.high_len == r.occurrences
    return r


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 8, 10, 13, 21, 31, 32])
def test_small_and_large_k(counter, k):
    rnd = random.Random(k)
    g = "".join(rnd.choice("ACGT") for _ in range(20_000))
    seqs = [g[i:i + 150] for i in (rnd.randrange(len(g) - 150) for _ in range(3000))] + ["ACGTN" * 20, "A" * 400, "T" * 60]
    fq = _fastq(seqs)
    for mc in (1, 2):
        r = _check(counter, fq, k, mc, bloom=True, memory_gb=1)
        assert r.smem_passes == 1 and r.smem_fallbacks == 0


@pytest.mark.parametrize("prefix,n,fallback", [(4, 60_000, False), (9, 60_000, False), (11, 30_000, False),
                                               (12, 40_000, True), (14, 60_000, True)])
@pytest.mark.parametrize("shape", [1, 2])
def test_many_kmers_of_one_prefix(counter, prefix, n, fallback, shape):
    """n distinct k-mers that start with the same `prefix` bases, some of them
    repeated: too many for one sub-bucket's table.  Sub-buckets and rounds
    tell at most 13 bases apart (8 + 12 + 6 bits), so 12 shared bases leave 4
    ranges of 10000 k-mers, more than a table has slots."""
    rnd = random.Random(prefix)
    k = 31
    p = "AC" + "".join(rnd.choice("ACGT") for _ in range(prefix - 2))
    # first base A, last base A: the forward strand is the canonical one
    seqs = list({p + "".join(rnd.choice("ACGT") for _ in range(k - prefix - 1)) + "A" for _ in range(n)})
    seqs += [seqs[i % 777] for i in range(5000)] + ["".join(rnd.choice("ACGT") for _ in range(150)) for _ in range(200)]
    rnd.shuffle(seqs)
    counter.set_tuning(count_shape=shape)
    for mc in (1, 2):
        r = _check(counter, _fastq(seqs), k, mc, bloom=True, memory_gb=1)
        assert (r.smem_fallbacks > 0) == fallback and r.smem_passes == (0 if fallback else 1)
    counter.set_tuning(count_shape=1)


def test_one_kmer_of_many_occurrences(counter):
    """Poly-A reads: one sub-bucket holds a few million equal keys."""
    rnd = random.Random(1)
    seqs = ["A" * 5000] * 500 + ["".join(rnd.choice("ACGT") for _ in range(150)) for _ in range(20_000)]
    rnd.shuffle(seqs)
    fq = _fastq(seqs)
    assert len(fq) > 4 << 20
    _check(counter, fq, 31)              # a plain job on the prefix path
    _check(counter, fq, 31, 2, bloom=True, memory_gb=1)


@pytest.mark.parametrize("per_bucket", [900, 1100, 2100, 4200, 8100, 16500])
def test_sort_units_of_every_size(counter, per_bucket):
    """Distinct k-mers spread over the buckets: records per unit on both sides
    of each size class's edge."""
    rng = np.random.default_rng(per_bucket)
    bases = np.frombuffer(b"ACGT", np.uint8)
    reads = bases[rng.integers(0, 4, size=(per_bucket * 256 // 118, 150))]
    fq = b"".join(b"@r\n" + r.tobytes() + b"\n+\n" + b"I" * 150 + b"\n" for r in reads)
    _check(counter, fq, 31, 1, bloom=True, memory_gb=1)


@pytest.mark.parametrize("n", [1, 3, 1023, 4095, 4096, 4097, 8193])
@pytest.mark.parametrize("k", [31, 47])
def test_queries_at_chunk_edges(counter, n, k):
    """n records around the selection's chunks (4096 counts, four per load),
    with 1, 2 or 3 occurrences: top-N of several N and the count <= 2 set."""
    rnd = random.Random(n)
    g = "".join(rnd.choice("ACGT") for _ in range(n + k - 1))
    kmers = [g[i:i + k] for i in range(n)]
    seqs = [g] + [kmers[i] for i in range(n) if i % 3 != 0] + [kmers[i] for i in range(n) if i % 7 == 1]
    fq = _fastq(seqs)
    want_k, want_c = (O.exact_records if k <= 32 else O.exact_records_wide)([fq], k, U32)
    assert len(want_c) == n
    order = np.argsort(-want_c.astype(np.int64), kind="stable")
    for top in (1, 7, n, n + 5):
        r = counter.count([fq], k=k, count_max=U32, top_n=top, want_le2=True)
        assert np.array_equal(r.top_keys, want_k[order[:top]]) and np.array_equal(r.top_counts, want_c[order[:top]])
        assert np.array_equal(r.le2_keys, want_k[want_c <= 2]) and np.array_equal(r.le2_counts, want_c[want_c <= 2])


def _wide_reads(seed, n, lo, hi, genome):
    rnd = random.Random(seed)
    g = "".join(rnd.choice("ACGT") for _ in range(genome))
    comp = str.maketrans("ACGT", "TGCA")
    seqs = []
    for _ in range(n):
        ln = rnd.randint(lo, hi)
        i = rnd.randrange(genome - ln)
        s = list(g[i:i + ln])
        for j in range(ln):
            if rnd.random() < 0.004:
                s[j] = rnd.choice("ACGTN")
        s = "".join(s)
        seqs.append(s.translate(comp)[::-1] if rnd.random() < 0.5 else s)
    return seqs


def _check_wide(c, files, k, min_count=1, **kw):
    all_k, all_c = O.exact_records_wide(files, k, U32)
    m = all_c >= min_count
    r = c.count(files, k=k, count_max=U32, min_count=min_count, hist_max=300, top_n=20, want_le2=True, **kw)
    assert np.array_equal(r.keys, all_k[m]) and np.array_equal(r.counts, all_c[m])
    assert r.hist.tolist() == O.histogram(all_c, 1, 300).tolist()
    assert r.distinct == len(all_k) and r.occurrences == int(all_c.sum(dtype=np.uint64))
    order = np.argsort(-all_c[m].astype(np.int64), kind="stable")[:20]
    assert np.array_equal(r.top_keys, all_k[m][order])
    return r


@pytest.mark.parametrize("k", [33, 34, 47, 48, 63, 64, 65, 66, 80, 95, 96, 97, 112, 127, 128])
def test_wide_kmers(counter, k):
    """Two- and four-word k-mers on the prefix path: every remainder of k at a
    word's edge, ragged reads of both strands with N bases in two files, long
    lines across tiles, palindromes."""
    seqs = _wide_reads(k, 14_000, 130, 250, 60_000)
    rnd = random.Random(5)
    half = "".join(rnd.choice("ACGT") for _ in range(70))
    pal = half + half.translate(str.maketrans("ACGT", "TGCA"))[::-1]
    seqs += [pal, pal, "A" * 300, "T" * 200, "".join(rnd.choice("ACGT") for _ in range(30_000))]
    rnd.shuffle(seqs)
    files = [_fastq(seqs[:9000]), _fastq(seqs[9000:])]
    assert sum(len(f) for f in files) > 4 << 20
    for mc in (1, 2):
        r = _check_wide(counter, files, k, mc)
        assert r.smem_passes == 1 and r.smem_fallbacks == 0


@pytest.mark.parametrize("k", [55, 101])
def test_wide_kmers_in_passes_and_shapes(counter, k):
    files = [_fastq(_wide_reads(k, 14_000, 140, 250, 400_000))]
    for shape in (1, 2):
        counter.set_tuning(count_shape=shape, scatter_shape=shape, sampled_region_keys=1)
        one = _check_wide(counter, files, k)
        many = _check_wide(counter, files, k, pass_bytes=32 << 20)
        assert one.passes == 1 and many.passes > 1 and many.smem_passes == many.passes
    counter.set_tuning(count_shape=1, scatter_shape=1, sampled_region_keys=64 << 20)


@pytest.mark.parametrize("k,prefix,fallback", [(63, 10, False), (63, 40, True), (127, 10, False), (127, 100, True)])
def test_many_wide_kmers_of_one_prefix(counter, k, prefix, fallback):
    rnd = random.Random(prefix)
    p = "AC" + "".join(rnd.choice("ACGT") for _ in range(prefix - 2))
    seqs = list({p + "".join(rnd.choice("ACGT") for _ in range(k - prefix - 1)) + "A" for _ in range(30_000)})
    seqs += [seqs[i % 777] for i in range(3000)] + ["".join(rnd.choice("ACGT") for _ in range(150)) for _ in range(2000)]
    rnd.shuffle(seqs)
    r = _check_wide(counter, [_fastq(seqs)], k)
    assert (r.smem_fallbacks > 0) == fallback and (r.smem_passes == 0) == fallback


def test_wide_table_full_once_is_cut_and_counted_again(counter):
    import ktcountermemorygreedy_b200 as kc
    files = [_fastq(_wide_reads(9, 14_000, 140, 250, 100_000))]
    for k in (31, 63, 127):
        check = _check_wide if k > 32 else lambda c, f, kk, **kw: _check(c, f[0], kk, **kw)
        check(counter, files, k, fault_inject=kc.INJECT_TABLE_FULL_ONCE)


def _check_batch(counter, samples, ks, **kw):
    fqs = [_fastq(s) for s in samples]
    rs = counter.count_batch([[f] for f in fqs], ks, count_max=U32, hist_max=9000, **kw)
    for f, k, r in zip(fqs, ks, rs):
        all_k, all_c = O.exact_records([f], k, U32)
        m = all_c >= kw.get("min_count", 1)
        assert np.array_equal(r.keys, all_k[m]) and np.array_equal(r.counts, all_c[m])
        assert r.hist.tolist() == O.histogram(all_c, 1, 9000).tolist()
        assert r.distinct == len(all_k) and r.occurrences == int(all_c.sum(dtype=np.uint64))
    return rs


@pytest.mark.parametrize("min_count", [1, 2])
@pytest.mark.parametrize("n", [1, 2, 255, 256, 257])
def test_batch_of_samples(counter, n, min_count):
    """Samples as buckets: every k, up to and beyond the samples of one pass,
    empty samples, samples without a window of k bases, several tiles long,
    and k-mers with more occurrences than the dense histogram holds (the list
    then carries the sample) in the first and the last sample."""
    rnd = random.Random(n)
    g = "".join(rnd.choice("ACGT") for _ in range(4000))
    samples = []
    for i in range(n):
        reads = [g[j:j + 120] for j in (rnd.randrange(len(g) - 120) for _ in range(rnd.choice((0, 1, 5, 200))))]
        samples.append(reads + ["ACGTN" * 3, "C" * 40] if i % 5 else reads)
    samples[0] = samples[0] + ["A" * 5000, "T" * 300]
    samples[-1] = samples[-1] + ["AC" * 2500]
    rs = _check_batch(counter, samples, [1 + (7 * i + n) % 32 for i in range(n)], min_count=min_count)
    assert all(r.smem_passes == 1 and r.smem_fallbacks == 0 for r in rs)


@pytest.mark.parametrize("prefix,fallback", [(3, False), (7, False), (11, True)])
def test_batch_sample_of_one_prefix(counter, prefix, fallback):
    """One sample's k-mers share their first bases: sub-buckets and rounds tell
    at most 9 bases apart, so 11 leave one range of all k-mers, and the whole
    batch is counted in global-memory tables."""
    rnd = random.Random(prefix)
    p = "AC" + "".join(rnd.choice("ACGT") for _ in range(prefix - 2))
    skew = list({p + "".join(rnd.choice("ACGT") for _ in range(30 - prefix)) + "A" for _ in range(60_000)})
    plain = ["".join(rnd.choice("ACGT") for _ in range(150)) for _ in range(300)]
    rs = _check_batch(counter, [plain, skew + skew[:999], plain[:50]], [21, 31, 32])
    assert all((r.smem_fallbacks > 0) == fallback and r.smem_passes == (0 if fallback else 1) for r in rs)


@pytest.mark.parametrize("tiles", [1, 2, 2047, 2048, 2049, 16384, 16385])
def test_line_numbers_at_scan_edges(counter, tiles):
    """One record per 8 KiB tile, tile counts at the edges of one scan block and
    of the one-launch scan: a wrong line number would count the quality lines
    (letters) too."""
    n = (8192 - 7) // 2
    rec = b"@r\n" + b"A" * n + b"\n+\n" + b"C" * n + b"\n"
    fq = (b"@" + b"r" * (8192 - len(rec) + 1) + rec[2:]) * tiles
    assert len(fq) == 8192 * tiles
    for bloom in (False, True):
        r = counter.count([fq], k=31, count_max=U32, hist_max=10, **(dict(bloom=True, memory_gb=1) if bloom else {}))
        assert r.occurrences == (n - 30) * tiles and r.distinct == 1
        assert r.keys.tolist() == [0] and r.counts.tolist() == [(n - 30) * tiles]


@pytest.mark.parametrize("k,same", [(33, 20), (63, 31), (63, 33), (64, 60), (65, 40), (96, 64), (127, 70), (127, 100), (128, 124)])
def test_wide_runs_that_start_alike(counter, k, same):
    """Runs of k-mers with the same first `same` bases, told apart by any later
    word: every place of a run's first difference, between the words too."""
    rnd = random.Random(k + same)
    seqs = []
    for _ in range(300):
        p = "A" + "".join(rnd.choice("ACGT") for _ in range(same - 1))
        for _ in range(rnd.choice((1, 2, 3, 17, 40))):
            seqs.append(p + "".join(rnd.choice("ACGT") for _ in range(k - same - 1)) + "A")
    seqs += seqs[::3]
    f = _fastq(seqs)
    all_k, all_c = O.exact_records_wide([f], k)
    r = counter.count([f], k=k, count_max=U32)
    assert r.smem_passes == 1
    assert np.array_equal(r.keys, all_k) and np.array_equal(r.counts, all_c)


@pytest.mark.parametrize("top_n", [1, 65_535, 65_536, 65_537, 90_000, 200_000])
def test_top_n_on_both_sides_of_one_wait(counter, top_n):
    """Top-N lists up to 65536 come back with their lengths, longer ones after
    them; lists shorter than N (fewer records) too."""
    rng = np.random.default_rng(5)
    bases = np.frombuffer(b"ACGT", np.uint8)
    reads = bases[rng.integers(0, 4, size=(900, 150))]
    fq = b"".join(b"@r\n" + r.tobytes() + b"\n+\n" + b"I" * 150 + b"\n" for i, r in enumerate(reads) for _ in range(1 + i % 3))
    all_k, all_c = O.exact_records([fq], 31, U32)
    assert 100_000 < len(all_c) < 200_000
    order = np.argsort(-all_c.astype(np.int64), kind="stable")[:top_n]
    r = counter.count([fq], k=31, count_max=U32, top_n=top_n)
    assert np.array_equal(r.top_keys, all_k[order]) and np.array_equal(r.top_counts, all_c[order])
