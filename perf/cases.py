"""The work that users of this package have it do, as timed cases.

A case is a dict of plain values; ``prepare`` makes what a program has in hand
before the call, ``run`` makes one call through the package's public entry
points and returns its whole outputs, ``work`` says what a call cannot do
without, ``exact`` gives the outputs as plain torch and numpy compute them.

The inputs are synthetic FASTQ of the workloads' shapes
(``ktcountermemorygreedy_b200.synth``): reads from uniform positions on either
strand of a random genome (5% repeat families above 20 Mbp, as in the single
large job), substitution errors, optional N bases.  Every kind of call is
listed at one or more sizes of its range; ``draw`` spreads over the ranges.

kind      what it stands for
job       one counting job on reads: histogram and the 1000 most frequent k-mers
          (the served request's and the benchmark's outputs)
contigs   one counting job on an assembly: the sorted exact records + histogram
batch     many samples of a sequencing run in one batched job, their histograms
merge     histogram_tool / dump_tool on a tmp_dir of the reference's counter
dump      the sorted text dump of a job's records
"""
from __future__ import annotations

import math

import numpy as np
import torch

import ktcountermemorygreedy_b200 as kc
from ktcountermemorygreedy_b200 import synth

U32 = kc.U32_MAX
_counter = None


def counter():
    """The handle a program opens once: one job on the device at a time."""
    global _counter
    if _counter is None:
        _counter = kc.KmerCounter(max_inflight_jobs=1)
    return _counter


def job(name, reads, genome, k, **kw):
    c = dict(kind="job", reads=reads, genome=genome, k=k, len_min=150, len_max=150, sub=0.01, n_rate=0.0, files=1,
             resident=False, bloom=False, memory_gb=64, min_count=1, top_n=1000, want_le2=False, keep_records=False)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def contigs(name, n, genome, k, **kw):
    """The consensus sequences of an assembly as FASTQ; its k-mers (k >= 29)
    are distinct, so another seed's records are as many."""
    c = dict(kind="contigs", contigs=n, genome=genome, k=k, resident=False, bloom=False, memory_gb=64, min_count=1,
             top_n=0, want_le2=False, keep_records=True)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the records of a viral consensus: a call so small that launches and
        # read-backs are all there is
        contigs("virus_30kb_k31", 1, 30_000, 31),
        # a served request of the median size: histogram and top-1000 of 200k
        # reads from a 50 Mbp genome, from host memory
        job("request_200k_k25", 200_000, 50_000_000, 25),
        # every k-mer of a 20 Mbp assembly, the records back in host memory
        contigs("assembly_20M_k31", 57, 20_000_000, 31),
        # every k-mer of a 20 Mbp genome's reads at 30x (kmer_counter's own
        # settings: no Bloom split, min count 1), the reads on the device
        job("plain_4M_k31", 4_000_000, 20_000_000, 31, resident=True),
        # the same reads through the Bloom split from host memory: the upload
        # streamed under the counting
        job("bloom_host_4M_k31", 4_000_000, 20_000_000, 31, bloom=True, min_count=2),
        # the single large job (100 Mbp, 30x, the benchmark's workload)
        job("bloom_20M_k31", 20_000_000, 100_000_000, 31, bloom=True, min_count=2, resident=True),
        # Bloom split with the k-mers seen once kept as records: ragged reads
        # with N bases in two files (paired ends)
        job("bloom_all_1M_k21", 1_000_001, 15_000_000, 21, bloom=True, resident=True, len_min=76, len_max=151,
            n_rate=0.001, files=2),
        # two- and four-word k-mers for assembly graphs
        job("wide_2M_k63", 2_000_000, 10_000_000, 63, min_count=2, resident=True),
        job("wide_500k_k127", 500_003, 5_000_000, 127, resident=True, len_min=140, len_max=250),
        # a plate of samples of uneven depth in one batch, k = 21 and 31
        dict(name="batch_48", kind="batch", samples=48, reads_min=2_000, reads_max=60_000, genome=20_000_000, len_min=100,
             len_max=250, sub=0.01, k=21, k_odd=31),
        # the precise merge of counted (high) and once-seen (low) k-mers
        dict(name="merge_2M_8M_k31", kind="merge", high=2_000_000, low=8_000_000, k=31, count_max=255),
        # 2M records to the sorted text dump
        dict(name="dump_2M_k31", kind="dump", records=2_000_000, k=31),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "bloom", "bloom", "bloom_all", "request", "contigs", "contigs", "wide", "wide", "batch",
                       "merge", "dump"])
    if kind == "batch":
        lo = _log(rng, 200, 5_000)
        return dict(kind="batch", samples=rng.randint(3, 64), reads_min=lo, reads_max=lo * rng.randint(2, 20),
                    genome=_log(rng, 1_000_000, 30_000_000), len_min=rng.randint(75, 120), len_max=rng.randint(121, 250),
                    sub=rng.uniform(0.002, 0.02), k=rng.randint(15, 25), k_odd=rng.randint(26, 32))
    if kind == "merge":
        return dict(kind="merge", high=_log(rng, 10_000, 4_000_000), low=_log(rng, 10_000, 10_000_000),
                    k=rng.randint(27, 31), count_max=rng.choice([255, 1000, 65535]))
    if kind == "dump":
        return dict(kind="dump", records=_log(rng, 10_000, 4_000_000), k=rng.choice([17, 21, 25, 31, 32]))
    if kind == "contigs":
        g = _log(rng, 10_000, 30_000_000)
        return contigs(None, rng.randint(1, 60), g, rng.choice([29, 31, 31, 32, 63, 127]), resident=rng.random() < 0.5,
                       bloom=rng.random() < 0.3, want_le2=rng.random() < 0.3)
    lo = rng.randint(75, 150)
    hi = lo if rng.random() < 0.5 else rng.randint(lo, 250)
    c = dict(len_min=lo, len_max=hi, sub=rng.uniform(0.002, 0.02), n_rate=rng.choice([0.0, 0.0, 0.001]),
             resident=rng.random() < 0.5, files=rng.choice([1, 1, 2]))
    if kind == "wide":
        k = rng.choice([33, 47, 55, 63, 64, 77, 95, 111, 127, 128])
        n = _log(rng, 5_000, 1_000_000)
        c.update(len_min=max(lo, k + 60), len_max=max(hi, k + 60), min_count=rng.choice([1, 2]))
    elif kind == "request":
        k, n = rng.choice([21, 25, 31]), _log(rng, 5_000, 1_000_000)
    elif kind == "plain":
        k, n = rng.choice([15, 17, 21, 25, 27, 31, 32]), _log(rng, 500, 2_000_000)
    elif kind == "bloom":
        k, n = rng.choice([17, 21, 25, 27, 31, 32]), _log(rng, 10_000, 6_000_000)
        c.update(bloom=True, min_count=2, memory_gb=rng.choice([8, 16, 64]))
    else:
        k, n = rng.choice([19, 21, 25, 31]), _log(rng, 10_000, 2_000_000)
        c.update(bloom=True, memory_gb=rng.choice([8, 16, 64]))
    genome = max(10_000, int(n * (c["len_min"] + c["len_max"]) / 2 / rng.uniform(5, 60)))
    return job(None, n, genome, k, **c)


# ---- inputs ------------------------------------------------------------------

class Resident:
    """FASTQ on the device (kc_input_upload), given back with its last use."""

    def __init__(self, files):
        self.counter = counter()
        self.input = self.counter.upload(files)

    def __del__(self):
        try:
            self.counter.free_input(self.input)
        except Exception:
            pass


def _genome(seed, length):
    if length >= 20_000_000:
        return synth.genome(seed, length, 0.05, 200, (1000, 5000), (10, 500), 0.02)
    return synth.genome(seed, length)


def _pinned(n):
    """Page-locked host memory, a reader's buffer."""
    if torch.cuda.is_available():
        return torch.empty(max(n, 1), dtype=torch.uint8, pin_memory=True).numpy()
    return np.empty(max(n, 1), np.uint8)


def _contigs(case, seed, pinned):
    """The genome cut at random places, one FASTQ record a piece."""
    g = synth.genome(seed, case["genome"])
    rng = np.random.default_rng(seed)
    cuts = np.sort(rng.choice(np.arange(1, len(g) // 200), case["contigs"] - 1, replace=False)) * 200
    parts = []
    for i, piece in enumerate(np.split(g, cuts)):
        parts += [np.frombuffer(b"@contig%03d\n" % i, np.uint8), piece, np.frombuffer(b"\n+\n", np.uint8),
                  np.full(len(piece), 73, np.uint8), np.frombuffer(b"\n", np.uint8)]
    buf = (_pinned if pinned else lambda n: np.empty(n, np.uint8))(sum(len(p) for p in parts))
    return np.concatenate(parts, out=buf)


def _fastq(case, seed, pinned=False):
    """The case's files, one FASTQ buffer each."""
    if case["kind"] == "contigs":
        return [_contigs(case, seed, pinned)]
    g = _genome(seed, case["genome"])
    lens = (case["len_min"], case["len_max"])
    n, out = case["reads"], []
    for f in range(case["files"]):
        m = n // case["files"] + (1 if f < n % case["files"] else 0)
        buf = _pinned(synth.reads_size(seed + f, m, lens)) if pinned else None
        out.append(synth.reads(g, seed + f, m, lens, case["sub"], case["n_rate"], out=buf))
    return out


def _random_kmers(gen, n, k, dev):
    """n distinct canonical k-mers (k <= 31) in random order, as r words."""
    top = (1 << (2 * k)) - 1
    s = torch.randint(0, top + 1, (int(n * 1.02) + 64,), generator=gen, device=dev, dtype=torch.int64)
    r, s = _canonical(_pair_reverse(s, k), s, k)
    u = torch.unique(r)
    return u[torch.randperm(u.numel(), generator=gen, device=dev)[:n]]


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def prepare(case, seed):
    seed = int(seed) % (1 << 40) + 1
    st = dict(case=case)
    kind = case["kind"]
    if kind in ("job", "contigs"):
        files = _fastq(case, seed, pinned=not case["resident"])
        if case["resident"]:
            st["resident"] = Resident(files)
        else:
            st["files"] = files
        counter()
    elif kind == "batch":
        rng = np.random.default_rng(seed)
        n = np.exp(rng.uniform(math.log(case["reads_min"]), math.log(case["reads_max"]), case["samples"])).astype(int)
        st["samples"], st["ks"] = [], []
        for i, m in enumerate(n):
            g = synth.genome(seed * 1000 + i, case["genome"])
            lens = (case["len_min"], case["len_max"])
            buf = _pinned(synth.reads_size(seed * 1000 + i, int(m), lens))
            st["samples"].append([synth.reads(g, seed * 1000 + i, int(m), lens, case["sub"], 0.0, out=buf)])
            st["ks"].append(case["k"] if i % 2 == 0 else case["k_odd"])
        counter()
    elif kind == "merge":
        gen = torch.Generator(_dev()).manual_seed(seed)
        k, h, lo = case["k"], case["high"], case["low"]
        r = _random_kmers(gen, h + lo, k, _dev())
        h = min(h, max(1, r.numel() // 2))
        high, low = r[:h], r[h:]
        # a tenth of the low k-mers are in the high file too (the first
        # occurrence of a counted k-mer)
        both = min(high.numel(), low.numel() // 10)
        low = torch.cat([low[both:], high[:both]])
        low = low[torch.randperm(low.numel(), generator=gen, device=low.device)]
        counts = torch.randint(1, 60, (h,), generator=gen, device=high.device, dtype=torch.int64)
        counts[:: 997] = case["count_max"]
        st["high"], st["low"] = _words(high, k), _words(low, k)
        st["counts"] = counts.to(torch.int64).cpu().numpy().astype(np.uint32)
    else:
        rng = np.random.default_rng(seed)
        k, n = case["k"], case["records"]
        s = np.sort(rng.integers(0, 1 << 63, n, dtype=np.uint64) >> np.uint64(max(0, 63 - 2 * k)))
        st["keys"] = _np_words(s, k)
        # the same counts in another order for every seed: texts of one length
        st["counts"] = rng.permutation(np.minimum(np.random.default_rng(0).geometric(0.04, n), 255).astype(np.uint32))
    return st


def _job_args(case):
    return dict(k=case["k"], count_max=U32, bloom=case["bloom"], memory_gb=case["memory_gb"],
                min_count=case["min_count"], hist_min=1, hist_max=10000, top_n=case["top_n"],
                want_le2=case["want_le2"], keep_records=case["keep_records"])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("job", "contigs"):
        if "resident" in state:
            r = counter().count(input=state["resident"].input, copy=False, **_job_args(case))
        else:
            r = counter().count(state["files"], copy=False, **_job_args(case))
        return dict(keys=r.keys, counts=r.counts, hist=r.hist, top_keys=r.top_keys, top_counts=r.top_counts,
                    le2_keys=r.le2_keys, le2_counts=r.le2_counts, occurrences=int(r.occurrences),
                    distinct=int(r.distinct))
    if kind == "batch":
        rs = counter().count_batch(state["samples"], state["ks"], copy=False, count_max=U32, min_count=1, hist_min=1,
                                   hist_max=4095, keep_records=False)
        return dict(hist=np.array([r.hist for r in rs]),
                    totals=np.array([(r.occurrences, r.distinct) for r in rs], np.int64))
    if kind == "merge":
        k, c, h = kc.merge_records(state["high"], state["counts"], state["low"], case["k"], case["count_max"])
        return dict(keys=k, counts=c, hist=h)
    return np.frombuffer(kc.dump_bytes(state["keys"], state["counts"], case["k"]), np.uint8)


# ---- what a call cannot do without ----------------------------------------------

def _job_records(case):
    """Expected distinct k-mers and records of a job (uniform reads)."""
    k = case["k"]
    if case["kind"] == "contigs":
        n = case["genome"] - case["contigs"] * (k - 1)
        return n, n, n
    ln = (case["len_min"] + case["len_max"]) / 2
    occ = case["reads"] * max(ln - k + 1, 0)
    ok = (1 - case["sub"] - case["n_rate"]) ** k
    g = max(case["genome"], 1)
    cov = occ * ok / g
    genomic = g * (1 - math.exp(-cov))
    errors = occ * (1 - ok)
    repeated = g * (1 - math.exp(-cov) * (1 + cov))
    return occ, genomic + errors, repeated if case["min_count"] >= 2 else genomic + errors


def work(case):
    kind = case["kind"]
    if kind in ("job", "contigs"):
        if kind == "contigs":
            fastq = 2 * case["genome"] + 15 * case["contigs"]
        else:
            fastq = case["reads"] * (case["len_min"] + case["len_max"] + 6 + math.log10(max(case["reads"], 10)))
        _, distinct, records = _job_records(case)
        words = kc.key_words(case["k"])
        out = records * (8 * words + 4) if case["keep_records"] else 0
        if case["want_le2"]:
            out += distinct * (8 * words + 4)
        return dict(bytes=fastq + out + 80_000, flops=0)
    if kind == "batch":
        a, b = case["reads_min"], case["reads_max"]
        reads = case["samples"] * (b - a) / math.log(b / a)
        ln = (case["len_min"] + case["len_max"]) / 2
        return dict(bytes=reads * (2 * ln + 10) + case["samples"] * 4095 * 8, flops=0)
    if kind == "merge":
        return dict(bytes=case["high"] * 12 + case["low"] * 8 + (case["high"] + 0.9 * case["low"]) * 12 + 80_000,
                    flops=0)
    return dict(bytes=case["records"] * (12 + case["k"] + 4), flops=0)


# ---- the same outputs in plain torch and numpy -----------------------------------
#
# A k-mer (k <= 31) as two integers: s, its bases first-base-high (the printed
# order), and r, first-base-low; the package's word is r << (64 - 2k).  The
# reverse complement of (r, s) is (M - s, M - r) with M = 4^k - 1, and the
# canonical form is the one with the smaller r.

def _pair_reverse(s, k):
    r = torch.zeros_like(s)
    for i in range(k):
        r = (r << 2) | ((s >> (2 * i)) & 3)
    return r


def _canonical(r, s, k):
    m = (1 << (2 * k)) - 1
    fwd = r <= m - s
    return torch.where(fwd, r, m - s), torch.where(fwd, s, m - r)


def _words(r, k):
    return r.cpu().numpy().astype(np.uint64) << np.uint64(64 - 2 * k)


def _np_words(s, k):
    w = np.zeros_like(s)
    for i in range(k):
        w |= ((s >> np.uint64(2 * (k - 1 - i))) & np.uint64(3)) << np.uint64(64 - 2 * k + 2 * i)
    return w


def _extract(fastq, k):
    """(r, s) of every window of k valid bases in the sequence lines."""
    b = torch.from_numpy(np.ascontiguousarray(fastq)).to(_dev())
    nl = b == 10
    line = torch.cumsum(nl, 0) - nl.to(torch.int64)
    code = torch.full((256,), 4, dtype=torch.int64, device=b.device)
    for i, ch in enumerate("ACGT"):
        code[ord(ch)] = code[ord(ch.lower())] = i
    code[ord("U")] = code[ord("u")] = 3
    c = code[b.to(torch.int64)]
    c[(line & 3) != 1] = 4
    bad = torch.cumsum((c == 4).to(torch.int32), 0)
    n = c.numel() - k + 1
    if n <= 0:
        return c[:0], c[:0]
    first_bad = (c[:n] == 4).to(torch.int32)
    ok = (bad[k - 1:] - bad[:n] + first_bad) == 0
    at = torch.nonzero(ok).squeeze(1)
    r, s = torch.zeros_like(at), torch.zeros_like(at)
    for i in range(k):
        x = c[at + i]
        s = (s << 2) | x
        r |= x << (2 * i)
    return _canonical(r, s, k)


def _count(files, k, min_count, hist_max):
    rs = [_extract(f, k) for f in files]
    s = torch.cat([x[1] for x in rs])
    occ = s.numel()
    u, n = torch.unique(s, return_counts=True)
    hist = torch.bincount(n.clamp(max=hist_max + 1), minlength=hist_max + 2)[1:hist_max + 1]
    keep = n >= min_count
    return (_words(_pair_reverse(u[keep], k), k), n[keep].cpu().numpy().astype(np.uint32),
            hist.cpu().numpy().astype(np.int64), occ, int(u.numel()))


def exact(case, seed):
    """None above 31 bases (the two-integer form) and for large jobs."""
    seed = int(seed) % (1 << 40) + 1
    kind = case["kind"]
    if kind in ("job", "contigs"):
        if case["k"] > 31 or case.get("reads", 0) > 250_000:
            return None
        keys, counts, hist, occ, distinct = _count(_fastq(case, seed), case["k"], case["min_count"], 10000)
        e64, e32 = np.zeros(0, np.uint64), np.zeros(0, np.uint32)
        out = dict(keys=e64, counts=e32, hist=hist, top_keys=e64, top_counts=e32, le2_keys=e64, le2_counts=e32,
                   occurrences=occ, distinct=distinct)
        if case["top_n"]:
            best = np.argsort(-counts.astype(np.int64), kind="stable")[: case["top_n"]]
            out.update(top_keys=keys[best], top_counts=counts[best])
        if case["want_le2"]:
            out.update(le2_keys=keys[counts <= 2], le2_counts=counts[counts <= 2])
        if case["keep_records"]:
            out.update(keys=keys, counts=counts)
        return out
    if kind == "merge":
        st = prepare(case, seed - 1)
        k, w = case["k"], np.uint64(64 - 2 * case["k"])
        allk = torch.from_numpy((np.concatenate([st["high"], st["low"]]) >> w).astype(np.int64)).to(_dev())
        n = torch.from_numpy(np.concatenate([st["counts"].astype(np.int64), np.ones(len(st["low"]), np.int64)]))
        u, at = torch.unique(_pair_reverse(allk, k), return_inverse=True)
        c = torch.zeros(u.numel(), dtype=torch.int64, device=u.device).scatter_add_(0, at, n.to(u.device))
        c = c.clamp(max=case["count_max"])
        hist = torch.bincount(c, minlength=10001)[1:10001]
        return dict(keys=_words(_pair_reverse(u, k), k), counts=c.cpu().numpy().astype(np.uint32),
                    hist=hist.cpu().numpy().astype(np.int64))
    if kind == "dump" and case["records"] <= 300_000:
        st = prepare(case, seed - 1)
        return np.frombuffer("".join(f"{kc.kmer_string(int(w), case['k'])}\t{c}\n"
                                     for w, c in zip(st["keys"], st["counts"])).encode(), np.uint8)
    return None
