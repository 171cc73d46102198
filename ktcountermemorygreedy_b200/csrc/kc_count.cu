// kc_count.cu -- counting of k-mers by printed-order prefix, in shared memory,
// and the sort of the resulting records.
//
// The occurrences arrive partitioned twice, into 256 buckets by their first
// four bases and into sub-buckets by the next bases (launch_part by string,
// k_subpart_scatter), as string keys: the k bases first-base-high, left
// aligned, in one, two or four 64-bit words.  So the sub-buckets are consecutive ranges of the printed order:
// once every sub-bucket's distinct k-mers are counted and sorted on their own,
// all records are in order and no sort of the whole set is left.
//
// Placement only uses the keys' values, never the order in which occurrences
// arrive: every count is exact, and an occurrence is the FIRST of its k-mer
// (src/BloomFilter.h:233-273, the reference's singleton split) exactly when
// it claims the k-mer's slot, which is the split a filter without false
// positives makes.
//
// Against the path it replaced (filter slices and 4096-slot tables per
// sub-bucket of an XXH3 partition, global bucket tables for plain jobs, and a
// sort of all records), on a B200: 20M reads (2.4G k-mers, 115M records,
// min count 2) count 27.1 -> 14.5 ms and sort 7.1 -> 1.1 ms; 4M reads with
// every k-mer kept (480M k-mers, 145M records) insert + compaction 11.8 ms ->
// scatter + count 5.0 ms, sort 11.8 -> 1.6 ms.
// k > 32, against an N-word table in HBM probed straight from the extraction and
// one stable LSD sort per word: 2M reads at k = 63 (176M k-mers, min count 2) scan,
// insert, compaction and sort 26.2 ms -> census, partition, scatter, count and sort
// 6.0 ms; 500k reads at k = 127 (29M records) 25.8 -> 4.2 ms.
#include <algorithm>

#include "kc_device.cuh"
#include "kc_kernels.cuh"

namespace kc {

namespace {

constexpr uint32_t FULLW = 0xffffffffu;
constexpr uint32_t CP_HIST = 512;           // counts below this are histogrammed in shared memory
constexpr uint32_t CP_QUEUE = 64;           // keys a warp has waiting for their next probe

__device__ __forceinline__ uint32_t lanes_below()
{
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

template <uint32_t N>
struct KeyN {
    unsigned long long w[N];
    __device__ __forceinline__ bool operator==(const KeyN &o) const
    {
        bool e = w[0] == o.w[0];
#pragma unroll
        for (uint32_t i = 1; i < N; ++i) e = e && w[i] == o.w[i];
        return e;
    }
};

// Key i of an array of N-word keys: one 8- or 16-byte access per word (pair).
template <uint32_t N, class INDEX, class LOAD>
__device__ __forceinline__ KeyN<N> load_key(const unsigned long long *p, INDEX i, LOAD load)
{
    KeyN<N> k;
    if constexpr (N == 1) {
        k.w[0] = load(p + i);
    } else {
        const ulonglong2 *q = reinterpret_cast<const ulonglong2 *>(p + i * N);
#pragma unroll
        for (uint32_t j = 0; j < N / 2; ++j) {
            const ulonglong2 v = load(q + j);
            k.w[2 * j] = v.x;
            k.w[2 * j + 1] = v.y;
        }
    }
    return k;
}

template <uint32_t N, class INDEX>
__device__ __forceinline__ void store_key(unsigned long long *p, INDEX i, const KeyN<N> &k)
{
    if constexpr (N == 1) {
        p[i] = k.w[0];
    } else {
        ulonglong2 *q = reinterpret_cast<ulonglong2 *>(p + i * N);
#pragma unroll
        for (uint32_t j = 0; j < N / 2; ++j) q[j] = make_ulonglong2(k.w[2 * j], k.w[2 * j + 1]);
    }
}

struct LoadStream {
    template <class T>
    __device__ __forceinline__ T operator()(const T *p) const { return __ldcs(p); }
};
struct LoadL2 {
    template <class T>
    __device__ __forceinline__ T operator()(const T *p) const { return __ldcg(p); }
};
struct LoadPlain {
    template <class T>
    __device__ __forceinline__ T operator()(const T *p) const { return *p; }
};

// Placement hash of a key: two 32-bit multiplies over its halves (the top
// bits are the same for a whole sub-bucket, so the low half leads), two more
// per further word.  The top bits are its home slot, an odd number from the
// next ones its probe step.  It never affects a count.
template <uint32_t N>
__device__ __forceinline__ uint32_t mix_of(const KeyN<N> &k)
{
    uint32_t h = 0;
#pragma unroll
    for (uint32_t i = N - 1; i > 0; --i)
        h = ((h ^ (uint32_t)k.w[i]) * 0x9E3779B1u + (uint32_t)(k.w[i] >> 32)) * 0xC2B2AE3Du;
    return ((h ^ (uint32_t)k.w[0]) * 0x9E3779B1u + (uint32_t)(k.w[0] >> 32)) * 0x85EBCA77u;
}

// Slots of two- and four-word keys: the count word says what state a slot is
// in.  A slot is claimed by one CAS of that word, its key written and then
// published; another thread compares keys only in published slots, and meets a
// claimed one again at its next probe step.
constexpr uint32_t SLOT_CLAIMED = 1u << 31, SLOT_PUBLISHED = 1u << 30, SLOT_COUNT = SLOT_PUBLISHED - 1;

// Counts one sub-bucket per block at a time.  The keys are inserted into an
// open-addressing table in shared memory (a slot only changes from empty to a
// key, by CAS; no barrier between tiles): every key looks at its home slot,
// where most are found or find their place; the others wait in the warp's queue
// until there are 32 of them, so that a probe step (claim, count, or on to the
// next slot and back into the queue) has all lanes busy.  (Each lane stepping
// its own keys to the end left 16 of 32 lanes active and 198 warp instructions
// per 32 keys; with the queue 23 and 172.  A ring that refilled each idle lane
// at every step took 248: more bookkeeping than probing.)  A home slot found
// empty is claimed at once when most keys are distinct (25M k-mers 0.34 -> 0.32
// ms; no difference at 3.3 occurrences each).  Then one sweep lists the used
// slots and takes them 32 at a time, so that no lane handles an empty one (two
// slots to a lane, a third of them used, the sweep was a fourth of all
// instructions: 2.4G k-mers of the 20M-read job 15.8 -> 14.5 ms, 480M k-mers with
// every record kept 3.21 -> 2.95): it writes the kept records to the front of the
// sub-bucket's place in the record arrays, adds every count to the histogram and
// empties the table for the next sub-bucket.  Bound by instruction issue (72%)
// and shared-memory wavefronts (60%).
// A table that fills up (more distinct k-mers than it holds) is
// emptied and the sub-bucket counted in rounds over halves of its key range
// (quarters, ... at most SUB_MAX_ROUNDS), each round reading the keys again
// from L2; a round's records lie after the earlier rounds' ones, and are a
// sort unit of their own.  A sub-bucket that no number of rounds fits, or that
// would take one block too long, is listed with what is left of it (kc_crowd.cu
// counts that).  The next sub-bucket's first keys are loaded before
// the sweep.  Histogram and totals go to the sub-bucket's group.
template <uint32_t N, uint32_t THREADS, uint32_t BPSM, uint32_t TBITS>
__global__ void __launch_bounds__(THREADS, BPSM) k_count_prefix(PrefixCountArgs a)
{
    constexpr uint32_t SLOTS = 1u << TBITS, PER_THREAD = N == 1 ? 3 : 4 / N;   // keys whose home slots are read together
    constexpr uint32_t TILE_KEYS = THREADS * PER_THREAD, WARPS = THREADS / 32;
    extern __shared__ __align__(16) uint8_t cp_smem[];
    unsigned long long *s_tk = reinterpret_cast<unsigned long long *>(cp_smem);   // SLOTS keys
    uint32_t *s_tc = reinterpret_cast<uint32_t *>(s_tk + N * SLOTS);              // their counts (N > 1: and states)
    uint32_t *s_hist = s_tc + SLOTS;                                              // CP_HIST
    unsigned long long *q_key =                                                   // CP_QUEUE keys per warp
        reinterpret_cast<unsigned long long *>(s_hist + CP_HIST) + (threadIdx.x >> 5) * (CP_QUEUE * N);
    uint16_t *q_slot = reinterpret_cast<uint16_t *>(s_hist + CP_HIST + 2 * N * CP_QUEUE * WARPS) +
                       (threadIdx.x >> 5) * CP_QUEUE;
    __shared__ uint32_t s_out, s_full, s_next, s_next_n;
    __shared__ unsigned long long s_next_off, s_kept;   // s_kept, s_group: only thread 0 writes them
    __shared__ uint32_t s_group;
    __shared__ SubCfg s_cfg[2];   // this sub-bucket's and the next one's
    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t lt = lanes_below();
    // sub-buckets that outgrew their regions are incomplete: nothing is counted
    if (a.counters[C_REGION_OVF]) return;
    for (uint32_t i = tid; i < SLOTS; i += THREADS) {
        if (N == 1) s_tk[i] = EMPTY_KEY;
        s_tc[i] = 0;
    }
    for (uint32_t i = tid; i < CP_HIST; i += THREADS) s_hist[i] = 0;
    uint32_t n_distinct = 0, n_once = 0, n_one = 0;   // per lane and group: below 2^32 whatever the pass
    uint32_t rounds0 = 1, par = 1;
    // thread 0 takes the next sub-bucket while this one is counted
    auto take_next = [&]() {
        const uint32_t s = atomicAdd(a.next_sub, 1u);
        s_next = s;
        if (s < a.n_sub) {
            s_next_n = a.sub_count[s];
            s_next_off = a.sub_off[s];
            s_cfg[par ^ 1] = a.sc[a.sub_bucket[s]];
        }
    };
    if (tid == 0) {
        s_out = 0;
        s_full = 0;
        s_kept = 0;
        take_next();
        s_group = s_next < a.n_sub ? s_cfg[0].group : 0u;
    }
    __syncthreads();
    // the first tile of keys of a sub-bucket
    KeyN<N> kn[PER_THREAD];
    constexpr uint32_t STEP = N == 1 ? 32 : THREADS;
    const uint32_t first = N == 1 ? (uint32_t)(tid >> 5) * (32 * PER_THREAD) + (uint32_t)lane : (uint32_t)tid;
    auto load_first = [&](unsigned long long off, uint32_t cnt) {
#pragma unroll
        for (uint32_t r = 0; r < PER_THREAD; ++r)
            if (first + STEP * r < cnt) kn[r] = load_key<N>(a.keys, off + first + STEP * r, LoadStream());
    };
    uint32_t sub = s_next, n = 0;
    unsigned long long base = 0;
    par = 0;
    if (sub < a.n_sub) {
        n = s_next_n;
        base = s_next_off;
        load_first(base, n);
    }
    // a group's histogram and totals; the block starts over
    auto flush = [&]() {
        __syncthreads();
        const uint32_t group = s_group;
        unsigned long long *hist = a.hist + (unsigned long long)group * a.hist_bins;
        for (uint32_t i = tid; i < CP_HIST; i += THREADS)
            if (s_hist[i]) {
                atomicAdd(&hist[i], (unsigned long long)s_hist[i]);
                s_hist[i] = 0;
            }
        unsigned long long s[3] = {n_distinct, n_once, n_one};
#pragma unroll
        for (int j = 0; j < 3; ++j)
            for (int o = 16; o > 0; o >>= 1) s[j] += __shfl_down_sync(FULLW, s[j], o);
        if (lane == 0) {
            if (s[0]) atomicAdd(&a.totals[3ull * group], s[0]);
            if (s[1]) atomicAdd(&a.totals[3ull * group + 1], s[1]);
            if (s[2]) atomicAdd(&hist[1], s[2]);
        }
        n_distinct = n_once = n_one = 0;
        if (tid == 0) {
            if (s_kept) atomicAdd(&a.totals[3ull * group + 2], s_kept);
            s_kept = 0;
        }
    };
    while (sub < a.n_sub) {
        const SubCfg &cfg = s_cfg[par];
        if (cfg.group != s_group) {
            flush();
            __syncthreads();
            if (tid == 0) s_group = cfg.group;
        }
        __syncthreads();   // s_next* read by all; the table is empty
        if (tid == 0) take_next();
        // slots for twice the keys where that is less than the whole table
        uint32_t lg = n > 1 ? 33 - __clz(n - 1) : 1;
        lg = lg < 9 ? 9 : (lg > TBITS ? TBITS : lg);
        const uint32_t smask = (1u << lg) - 1, hsh = 32 - lg;
        uint32_t rounds = n > SUB_ROUNDS_KEYS ? 1 : rounds0, rd = 0, off = 0, most = 0;
        bool failed = false;
        static_assert(SUB_KEYS_CAP < SLOT_COUNT, "a count would run into the state bits");
        const bool too_many = n > a.max_keys;
        while (rd < rounds && !too_many) {
            const uint32_t rmask = rounds - 1;
            const int rsh = 64 - (int)cfg.plen - (31 - __clz(rounds));   // rounds == 1: unused
            const bool reread = rd > 0 || failed;
            // a warp takes at most this many probe steps (a table that is not
            // nearly full needs far fewer)
            uint32_t qn = 0, steps = 0, most_steps = 3 * (n / THREADS + 1) + 64;
            // one more probe of the last `m` queued keys (m <= 32); those that
            // meet another key stay queued at their next slot
            auto probe_queue = [&](uint32_t m) {
                __syncwarp();
                qn -= m;
                ++steps;
                KeyN<N> key;
                uint32_t slot = 0;
                bool wait = false;
                if (lane < (int)m) {
                    key = load_key<N>(q_key, qn + lane, LoadPlain());
                    slot = q_slot[qn + lane];
                    if constexpr (N == 1) {
                        unsigned long long cur = *(volatile unsigned long long *)&s_tk[slot];
                        if (cur == EMPTY_KEY) {
                            cur = atomicCAS(&s_tk[slot], EMPTY_KEY, key.w[0]);
                            if (cur == EMPTY_KEY) cur = key.w[0];   // claimed
                        }
                        wait = cur != key.w[0];
                        if (!wait) atomicAdd(&s_tc[slot], 1u);
                    } else {
                        uint32_t st = *(volatile uint32_t *)&s_tc[slot];
                        wait = true;
                        if (st == 0) {
                            st = atomicCAS(&s_tc[slot], 0u, SLOT_CLAIMED | 1u);
                            if (st == 0) {
                                volatile unsigned long long *d = s_tk + N * slot;
#pragma unroll
                                for (uint32_t j = 0; j < N; ++j) d[j] = key.w[j];
                                __threadfence_block();   // the key before the state
                                atomicOr(&s_tc[slot], SLOT_PUBLISHED);
                                wait = false;
                            }
                        }
                        if (st & SLOT_PUBLISHED) {
                            __threadfence_block();
                            if (load_key<N>(s_tk, slot, LoadPlain()) == key) {
                                atomicAdd(&s_tc[slot], 1u);
                                wait = false;
                            } else {
                                slot = (slot + (mix_of<N>(key) >> 3 | 1u)) & smask;
                            }
                        }
                    }
                }
                const uint32_t w = __ballot_sync(FULLW, wait);
                if (wait) {
                    const uint32_t at = qn + (uint32_t)__popc(w & lt);
                    store_key<N>(q_key, at, key);
                    q_slot[at] = (uint16_t)(N == 1 ? (slot + (mix_of<N>(key) >> 3 | 1u)) & smask : slot);
                }
                qn += (uint32_t)__popc(w);
                __syncwarp();
            };
            for (uint32_t t0 = first; t0 - (N == 1 ? (uint32_t)lane : (uint32_t)tid) < n; t0 += TILE_KEYS) {
                KeyN<N> k[PER_THREAD];
                bool in[PER_THREAD];
#pragma unroll
                for (uint32_t r = 0; r < PER_THREAD; ++r) in[r] = t0 + STEP * r < n;
                if (reread) {
#pragma unroll
                    for (uint32_t r = 0; r < PER_THREAD; ++r)
                        if (in[r]) k[r] = load_key<N>(a.keys, base + t0 + STEP * r, LoadL2());
                } else {
#pragma unroll
                    for (uint32_t r = 0; r < PER_THREAD; ++r) {
                        k[r] = kn[r];
                        const uint32_t i = t0 + TILE_KEYS + STEP * r;
                        if (i < n) kn[r] = load_key<N>(a.keys, base + i, LoadStream());
                    }
                }
                if (rounds > 1) {
#pragma unroll
                    for (uint32_t r = 0; r < PER_THREAD; ++r)
                        in[r] = in[r] && ((uint32_t)(k[r].w[0] >> rsh) & rmask) == rd;
                }
                // the home slots: most keys are there already and only counted
                uint32_t slot[PER_THREAD];
                bool hit[PER_THREAD];
                unsigned long long cur[PER_THREAD];
#pragma unroll
                for (uint32_t r = 0; r < PER_THREAD; ++r) {
                    slot[r] = mix_of<N>(k[r]) >> hsh;
                    if constexpr (N == 1) {
                        cur[r] = *(volatile unsigned long long *)&s_tk[slot[r]];
                    } else {
                        hit[r] = false;
                        if (in[r] && (*(volatile uint32_t *)&s_tc[slot[r]] & SLOT_PUBLISHED)) {
                            __threadfence_block();
                            hit[r] = load_key<N>(s_tk, slot[r], LoadPlain()) == k[r];
                        }
                    }
                }
                if constexpr (N == 1) {
#pragma unroll
                    for (uint32_t r = 0; r < PER_THREAD; ++r) {
                        if (in[r] && cur[r] == EMPTY_KEY) {
                            cur[r] = atomicCAS(&s_tk[slot[r]], EMPTY_KEY, k[r].w[0]);
                            if (cur[r] == EMPTY_KEY) cur[r] = k[r].w[0];
                        }
                        hit[r] = cur[r] == k[r].w[0];
                    }
                }
#pragma unroll
                for (uint32_t r = 0; r < PER_THREAD; ++r) {
                    if (in[r] && hit[r]) atomicAdd(&s_tc[slot[r]], 1u);
                    const bool wait = in[r] && !hit[r];
                    const uint32_t w = __ballot_sync(FULLW, wait);
                    if (wait) {
                        const uint32_t at = qn + (uint32_t)__popc(w & lt);
                        store_key<N>(q_key, at, k[r]);
                        q_slot[at] = (uint16_t)(N == 1 ? (slot[r] + (mix_of<N>(k[r]) >> 3 | 1u)) & smask : slot[r]);
                    }
                    qn += (uint32_t)__popc(w);
                    // below 32 again before the next keys come (the queue holds 64)
                    while (qn >= 32) {
                        if (steps > most_steps) {
                            qn = 0;   // full: counted again anyway
                            s_full = 1;
                        } else {
                            probe_queue(32);
                        }
                    }
                }
                if (__any_sync(FULLW, *(volatile uint32_t *)&s_full != 0)) break;
            }
            while (qn && steps <= most_steps) probe_queue(qn < 32 ? qn : 32);
            if (qn) s_full = 1;
            __syncthreads();
            if (s_full) {
                // emptied and counted again over half the range
                __syncthreads();
                for (uint32_t i = tid; i <= smask; i += THREADS) {
                    if (N == 1) s_tk[i] = EMPTY_KEY;
                    s_tc[i] = 0;
                }
                if (tid == 0) s_full = 0;
                __syncthreads();
                failed = true;
                rounds *= 2;
                rd *= 2;
                if (rounds > SUB_MAX_ROUNDS || n > SUB_ROUNDS_KEYS || rounds * n > SUB_MAX_READS ||
                    (int)cfg.plen + (31 - __clz(rounds)) > 64)
                    break;
                continue;
            }
            // the next sub-bucket's first keys arrive during the sweep
            if (rd + 1 == rounds) load_first(s_next_off, s_next < a.n_sub ? s_next_n : 0u);
            // the sweep: the used slots are listed (in the queue's memory, free
            // now), four per lane at a time, and taken 32 at once: records out,
            // histogram, slots emptied
            const unsigned long long out = base + off;
            const uint32_t cmax = cfg.count_max, keep_lo = cfg.min_count, keep_hi = cfg.max_count;
            uint16_t *used = reinterpret_cast<uint16_t *>(q_key);
            static_assert(CP_QUEUE * 8 * N / 2 >= 128 + 31, "a list of the slots of one step and the rest of the last");
            uint32_t un = 0;
            auto take_used = [&](uint32_t m) {
                __syncwarp();
                un -= m;
                uint32_t i = 0, c = 0;
                bool keep = false;
                KeyN<N> key;
                if (lane < (int)m) {
                    i = used[un + lane];
                    const uint32_t raw = N > 1 ? s_tc[i] & SLOT_COUNT : s_tc[i];
                    if constexpr (N == 1) key = load_key<N>(s_tk, i, LoadPlain());
                    s_tc[i] = 0;
                    if constexpr (N == 1) s_tk[i] = EMPTY_KEY;
                    ++n_distinct;
                    n_once += raw == 1;
                    c = raw < cmax ? raw : cmax;
                    if (c == 1) ++n_one;   // most k-mers of many inputs: one shared bin would serialize
                    else if (c < CP_HIST) atomicAdd(&s_hist[c], 1u);
                    else if (c < a.hist_bins) atomicAdd(&a.hist[(unsigned long long)s_group * a.hist_bins + c], 1ull);
                    else {
                        const unsigned long long q = atomicAdd(&a.counters[C_OVF_LEN], 1ull);
                        if (q >= a.ovf_cap) atomicOr(&a.counters[C_FLAGS], ERR_HIST_OVERFLOW_FULL);
                        else if (a.ovf64) a.ovf64[q] = ((unsigned long long)s_group << 32) | c;
                        else a.ovf[q] = c;
                    }
                    keep = c >= keep_lo && c <= keep_hi;
                }
                const uint32_t b = __ballot_sync(FULLW, keep);
                uint32_t at0 = 0;
                if (lane == 0) at0 = atomicAdd(&s_out, (m << 16) + (uint32_t)__popc(b));
                if (b) {
                    const uint32_t w = __shfl_sync(FULLW, at0, 0) & 0xFFFFu;
                    if (keep) {
                        const unsigned long long at = out + w + (uint32_t)__popc(b & lt);
                        if constexpr (N > 1) key = load_key<N>(s_tk, i, LoadPlain());
                        store_key<N>(a.rec_keys, at, key);
                        a.rec_counts[at] = c;
                    }
                }
                __syncwarp();
            };
            for (uint32_t i0 = 0; i0 <= smask; i0 += 4 * THREADS) {
                const uint32_t i = i0 + 4 * tid;
                uint4 c4 = make_uint4(0, 0, 0, 0);
                if (i <= smask) c4 = *reinterpret_cast<const uint4 *>(&s_tc[i]);
                const uint32_t b0 = __ballot_sync(FULLW, c4.x != 0), b1 = __ballot_sync(FULLW, c4.y != 0);
                const uint32_t b2 = __ballot_sync(FULLW, c4.z != 0), b3 = __ballot_sync(FULLW, c4.w != 0);
                uint32_t at = un + (uint32_t)(__popc(b0 & lt) + __popc(b1 & lt) + __popc(b2 & lt) + __popc(b3 & lt));
                if (c4.x) used[at++] = (uint16_t)i;
                if (c4.y) used[at++] = (uint16_t)(i + 1);
                if (c4.z) used[at++] = (uint16_t)(i + 2);
                if (c4.w) used[at] = (uint16_t)(i + 3);
                un += (uint32_t)(__popc(b0) + __popc(b1) + __popc(b2) + __popc(b3));
                while (un >= 32) take_used(32);
            }
            if (un) take_used(un);
            __syncthreads();
            static_assert(SLOTS < 65536, "a round's distinct k-mers and records in one word");
            const uint32_t len = s_out & 0xFFFFu, held = s_out >> 16;
            __syncthreads();
            if (tid == 0) {
                s_out = 0;
                if (len) {
                    constexpr uint32_t CAP0 = unit_cap0(N);
                    const uint32_t cls = len <= CAP0 ? 0 : (len <= 2 * CAP0 ? 1 : (len <= 4 * CAP0 ? 2 : 3));
                    const unsigned long long u = atomicAdd(&a.counters[C_UNITS + cls], 1ull);
                    if (u < a.lists.cap[cls]) a.units[a.lists.base[cls] + u] = SubUnit{sub, off, len, cfg.k};
                    else atomicOr(&a.counters[C_UNIT_OVF], 1ull);
                    s_kept += len;
                }
            }
            off += len;
            most = held > most ? held : most;
            ++rd;
        }
        const bool gave_up = rd < rounds;   // uniform
        if (tid == 0) {
            a.sub_len[sub] = off;
            if (gave_up) {
                const uint32_t b = a.sub_bucket[sub];
                atomicAdd(&a.counters[C_CROWD_KEYS], (unsigned long long)n);
                if (!too_many) {
                    atomicOr(&a.bucket_ovf[b], 1u);
                    atomicAdd(&a.counters[C_CROWD_TRIED], (unsigned long long)n);
                }
                a.crowd[atomicAdd(&a.counters[C_SUB_OVF], 1ull)] = CrowdSub{base, n, sub, off, rd, rounds, b};
            }
        }
        // sub-buckets are alike: the next one starts with as many rounds, or with
        // fewer when as large a share of its keys as were distinct here would
        // fill no more than 7/8 of a table in any of them (a table takes about
        // 94%, where a probe takes three steps on average).  Rounds that only
        // came down below a quarter of a table stayed at four for sub-buckets
        // of 8K to 16K distinct k-mers, which two hold.
        rounds0 = gave_up || !n ? 1u : rounds;
        while (rounds0 > 1 && (unsigned long long)most * rounds * s_next_n <=
                                  (unsigned long long)(SLOTS - SLOTS / 8) * (rounds0 / 2) * n)
            rounds0 /= 2;
        if (too_many) __syncthreads();   // thread 0 has taken the next sub-bucket
        if (gave_up) load_first(s_next_off, s_next < a.n_sub ? s_next_n : 0u);
        sub = s_next;
        n = s_next_n;
        base = s_next_off;
        par ^= 1;
    }
    flush();
}

// Sorts the records of one unit (a sub-bucket, or one round of it: at most
// CAP records of one range of the printed order) per block at a time and
// writes them, as k-mer words, to their final place.  The keys come into
// shared memory once; their indexes are placed by the 2^LGB values of the bits
// below the unit's common prefix (the xor of all its keys says in which word
// and where that ends), then each record finds its rank inside its run of a few
// records by comparing itself with the run's other keys: no lane waits for
// another, unlike an insertion sort per run.  A thread keeps its keys in
// registers up to the placing (read again from shared memory for both digits,
// 480M k-mers' 190M records took 1.74 ms, now 1.56); the ranking goes in placed
// order, so that records are written nearly in order.  Twice the digits took
// 1.65, 1024 threads 1.80.  The counts are read where they are written (a unit's
// counts stay in L1).  Bound by the shared-memory pipe.
template <uint32_t THREADS, uint32_t CAP, uint32_t LGB>
__global__ void __launch_bounds__(THREADS) k_unit_sort(const unsigned long long *tk, const uint32_t *tv,
                                                       const unsigned long long *sub_off,
                                                       const unsigned long long *sub_final, const SubUnit *units,
                                                       uint32_t n_units, unsigned long long *out_k, uint32_t *out_v,
                                                       uint64_t out_cap)
{
    constexpr uint32_t NB = 1u << LGB, PER = NB / THREADS, WARPS = THREADS / 32, OWN = CAP / THREADS;
    static_assert(NB % THREADS == 0 && CAP <= 65536, "layout");
    extern __shared__ __align__(16) uint8_t us_smem[];
    unsigned long long *s_keys = reinterpret_cast<unsigned long long *>(us_smem);   // CAP keys
    uint32_t *s_start = reinterpret_cast<uint32_t *>(s_keys + CAP);             // NB
    uint16_t *s_idx = reinterpret_cast<uint16_t *>(s_start + NB);                   // CAP
    __shared__ uint32_t s_warp[WARPS], s_xor[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (uint32_t ui = blockIdx.x; ui < n_units; ui += gridDim.x) {
        const SubUnit u = units[ui];
        const uint32_t m = u.len < CAP ? u.len : CAP;
        const unsigned long long src = sub_off[u.sub] + u.off, dst = sub_final[u.sub] + u.off;
        if (tid < 2) s_xor[tid] = 0;
#pragma unroll
        for (uint32_t j = 0; j < PER; ++j) s_start[j * THREADS + tid] = 0;
        __syncthreads();
        // common prefix: the bits in which no key differs from the first
        const unsigned long long k0 = tk[src];
        unsigned long long x = 0;
        unsigned long long key[OWN];
#pragma unroll
        for (uint32_t r = 0; r < OWN; ++r) {
            const uint32_t i = r * THREADS + tid;
            if (i < m) {
                key[r] = __ldcs(tk + src + i);
                s_keys[i] = key[r];
                x |= key[r] ^ k0;
            }
        }
        const uint32_t xh = __reduce_or_sync(FULLW, (uint32_t)(x >> 32)), xl = __reduce_or_sync(FULLW, (uint32_t)x);
        if (lane == 0) {
            if (xh) atomicOr(&s_xor[0], xh);
            if (xl) atomicOr(&s_xor[1], xl);
        }
        __syncthreads();
        const int pre = __clzll(((unsigned long long)s_xor[0] << 32) | s_xor[1]);   // 64: one record
        const int dsh = 64 - pre - (int)LGB > 0 ? 64 - pre - (int)LGB : 0;
        auto digit = [&](unsigned long long k) { return (uint32_t)(k >> dsh) & (NB - 1); };
#pragma unroll
        for (uint32_t r = 0; r < OWN; ++r)
            if (r * THREADS + tid < m) atomicAdd(&s_start[digit(key[r])], 1u);
        __syncthreads();
        // exclusive scan of the NB counts, PER consecutive ones per thread
        uint32_t c[PER], own = 0;
#pragma unroll
        for (uint32_t j = 0; j < PER; ++j) {
            c[j] = s_start[tid * PER + j];
            own += c[j];
        }
        uint32_t inc = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULLW, inc, o);
            if (lane >= o) inc += y;
        }
        if (lane == 31) s_warp[warp] = inc;
        __syncthreads();
        uint32_t run = inc - own;
#pragma unroll
        for (uint32_t w = 0; w < WARPS; ++w)
            if ((int)w < warp) run += s_warp[w];
#pragma unroll
        for (uint32_t j = 0; j < PER; ++j) {
            s_start[tid * PER + j] = run;
            run += c[j];
        }
        __syncthreads();
        // placing moves each start to its run's end: run d is [end of run d - 1, end of run d)
#pragma unroll
        for (uint32_t r = 0; r < OWN; ++r)
            if (r * THREADS + tid < m) s_idx[atomicAdd(&s_start[digit(key[r])], 1u)] = (uint16_t)(r * THREADS + tid);
        __syncthreads();
        for (uint32_t p = tid; p < m; p += THREADS) {
            const uint32_t i = s_idx[p];
            const unsigned long long key = s_keys[i];
            const uint32_t d = digit(key);
            const uint32_t lo = d ? s_start[d - 1] : 0u, hi = s_start[d];
            uint32_t rank = lo;
            for (uint32_t j = lo; j < hi; ++j) rank += s_keys[s_idx[j]] < key ? 1u : 0u;
            if (dst + rank < out_cap) {
                out_k[dst + rank] = pair_reverse(key >> (64 - 2 * u.k));
                out_v[dst + rank] = __ldg(&tv[src + i]);
            }
        }
        __syncthreads();
    }
}

// 1 if the N-word number at p, its words `stride` apart and the first the most
// significant, is less than o: the borrow of p - o.
template <uint32_t N>
__device__ __forceinline__ uint32_t words_less(const unsigned long long *p, uint32_t stride, const unsigned long long *o)
{
    uint32_t less;
    if constexpr (N == 2)
        asm("{ .reg .u64 t; sub.cc.u64 t, %1, %2; subc.cc.u64 t, %3, %4; subc.u32 %0, 0, 0; }"
            : "=r"(less)
            : "l"(p[stride]), "l"(o[1]), "l"(p[0]), "l"(o[0]));
    else
        asm("{ .reg .u64 t; sub.cc.u64 t, %1, %2; subc.cc.u64 t, %3, %4; subc.cc.u64 t, %5, %6; subc.cc.u64 t, %7, %8; "
            "subc.u32 %0, 0, 0; }"
            : "=r"(less)
            : "l"(p[3 * stride]), "l"(o[3]), "l"(p[2 * stride]), "l"(o[2]), "l"(p[stride]), "l"(o[1]), "l"(p[0]), "l"(o[0]));
    return less & 1u;
}

// The same for two- and four-word keys.  Word w of all keys lies together (keys
// side by side, 32 bytes apart, put the same word of eight of them in one bank:
// the shared-memory pipe was 90% busy, 60% of it conflicts).  Long k-mers of
// reads come in runs of ten and more that start alike (the same position with
// different errors further on): a run's records are compared whole, without
// branches, by lanes next to one another, which read the same record at a time.
// 29M 127-base k-mers of sequence covered 20 times 1.65 -> 1.03 ms (words apart
// alone 1.46, with comparisons that stopped at the first difference).
template <uint32_t N, uint32_t THREADS, uint32_t CAP, uint32_t LGB>
__global__ void __launch_bounds__(THREADS) k_unit_sort_wide(const unsigned long long *tk, const uint32_t *tv,
                                                            const unsigned long long *sub_off,
                                                            const unsigned long long *sub_final, const SubUnit *units,
                                                            uint32_t n_units, unsigned long long *out_k, uint32_t *out_v,
                                                            uint64_t out_cap)
{
    constexpr uint32_t NB = 1u << LGB, PER = NB / THREADS, WARPS = THREADS / 32, OWN = CAP / THREADS;
    static_assert(NB % THREADS == 0 && CAP % THREADS == 0 && CAP <= 65536, "layout");
    extern __shared__ __align__(16) uint8_t us_smem[];
    unsigned long long *s_keys = reinterpret_cast<unsigned long long *>(us_smem);   // N x CAP words
    uint32_t *s_start = reinterpret_cast<uint32_t *>(s_keys + N * CAP);             // NB
    uint16_t *s_idx = reinterpret_cast<uint16_t *>(s_start + NB);                   // CAP
    __shared__ uint32_t s_warp[WARPS], s_xor[2 * N];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (uint32_t ui = blockIdx.x; ui < n_units; ui += gridDim.x) {
        const SubUnit u = units[ui];
        const uint32_t m = u.len < CAP ? u.len : CAP;
        const unsigned long long src = sub_off[u.sub] + u.off, dst = sub_final[u.sub] + u.off;
        if (tid < 2 * (int)N) s_xor[tid] = 0;
#pragma unroll
        for (uint32_t j = 0; j < PER; ++j) s_start[j * THREADS + tid] = 0;
        __syncthreads();
        // common prefix: the bits in which no key differs from the first
        const KeyN<N> k0 = load_key<N>(tk, src, LoadPlain());
        unsigned long long x[N];
#pragma unroll
        for (uint32_t j = 0; j < N; ++j) x[j] = 0;
#pragma unroll
        for (uint32_t r = 0; r < OWN; ++r) {
            const uint32_t i = r * THREADS + tid;
            if (i < m) {
                const KeyN<N> key = load_key<N>(tk, src + i, LoadStream());
#pragma unroll
                for (uint32_t j = 0; j < N; ++j) {
                    s_keys[j * CAP + i] = key.w[j];
                    x[j] |= key.w[j] ^ k0.w[j];
                }
            }
        }
#pragma unroll
        for (uint32_t j = 0; j < N; ++j) {
            const uint32_t xh = __reduce_or_sync(FULLW, (uint32_t)(x[j] >> 32)), xl = __reduce_or_sync(FULLW, (uint32_t)x[j]);
            if (lane == 0) {
                if (xh) atomicOr(&s_xor[2 * j], xh);
                if (xl) atomicOr(&s_xor[2 * j + 1], xl);
            }
        }
        __syncthreads();
        // the first word in which keys differ, and the digit below its common bits
        uint32_t dw = 0;
        unsigned long long diff = 0;
#pragma unroll
        for (uint32_t j = 0; j < N; ++j)
            if (!diff) {
                diff = ((unsigned long long)s_xor[2 * j] << 32) | s_xor[2 * j + 1];
                dw = j;
            }
        const int pre = __clzll(diff);   // 64: one record
        const int dsh = 64 - pre - (int)LGB > 0 ? 64 - pre - (int)LGB : 0;
        const unsigned long long *s_dw = s_keys + dw * CAP;
        uint32_t d[OWN];
#pragma unroll
        for (uint32_t r = 0; r < OWN; ++r) {
            const uint32_t i = r * THREADS + tid;
            d[r] = 0;
            if (i < m) {
                d[r] = (uint32_t)(s_dw[i] >> dsh) & (NB - 1);
                atomicAdd(&s_start[d[r]], 1u);
            }
        }
        __syncthreads();
        // exclusive scan of the NB counts, PER consecutive ones per thread
        uint32_t c[PER], own = 0;
#pragma unroll
        for (uint32_t j = 0; j < PER; ++j) {
            c[j] = s_start[tid * PER + j];
            own += c[j];
        }
        uint32_t inc = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULLW, inc, o);
            if (lane >= o) inc += y;
        }
        if (lane == 31) s_warp[warp] = inc;
        __syncthreads();
        uint32_t run = inc - own;
#pragma unroll
        for (uint32_t w = 0; w < WARPS; ++w)
            if ((int)w < warp) run += s_warp[w];
#pragma unroll
        for (uint32_t j = 0; j < PER; ++j) {
            s_start[tid * PER + j] = run;
            run += c[j];
        }
        __syncthreads();
        // placing moves each start to its run's end: run d is [end of run d - 1, end of run d)
#pragma unroll
        for (uint32_t r = 0; r < OWN; ++r) {
            const uint32_t i = r * THREADS + tid;
            if (i < m) s_idx[atomicAdd(&s_start[d[r]], 1u)] = (uint16_t)i;
        }
        __syncthreads();
        for (uint32_t p = tid; p < m; p += THREADS) {
            const uint32_t i = s_idx[p], dg = (uint32_t)(s_dw[i] >> dsh) & (NB - 1);
            const uint32_t lo = dg ? s_start[dg - 1] : 0u, hi = s_start[dg];
            uint32_t rank = lo;
            if (hi - lo > 1) {
                unsigned long long own[N];
#pragma unroll
                for (uint32_t w = 0; w < N; ++w) own[w] = s_keys[w * CAP + i];
                for (uint32_t j = lo; j < hi; ++j) rank += words_less<N>(s_keys + s_idx[j], CAP, own);
            }
            if (dst + rank < out_cap) {
                // string order back to k-mer words: word w holds the 32 bases
                // ending 32w before the last, newest at the top
                KeyN<N> key;
#pragma unroll
                for (uint32_t w = 0; w < N; ++w) {
                    const int b = (int)u.k - 32 * (int)(w + 1);   // first base of the word
                    unsigned long long v = 0;
                    if (b >= 0) {
                        const uint32_t o = 2 * (b & 31);
                        const unsigned long long *q = s_keys + (uint32_t)(b >> 5) * CAP + i;
                        v = q[0] << o;
                        if (o) v |= q[CAP] >> (64 - o);
                    } else if (b > -32) {
                        v = s_keys[i] >> (-2 * b);
                    }
                    key.w[w] = pair_reverse(v);
                }
                store_key<N>(out_k, dst + rank, key);
                out_v[dst + rank] = __ldg(&tv[src + i]);
            }
        }
        __syncthreads();
    }
}

int n_sms()
{
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 148;
}

template <uint32_t N, uint32_t THREADS, uint32_t BPSM, uint32_t TBITS>
cudaError_t launch_count_prefix_t(const PrefixCountArgs &a, cudaStream_t st)
{
    const size_t smem = ((size_t)1 << TBITS) * (8 * N + 4) + CP_HIST * 4 + (THREADS / 32) * CP_QUEUE * (8 * N + 2);
    auto kern = k_count_prefix<N, THREADS, BPSM, TBITS>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    note_kernel_launch();
    kern<<<std::min<uint32_t>(a.n_sub, (uint32_t)n_sms() * BPSM), THREADS, smem, st>>>(a);
    return cudaGetLastError();
}

template <uint32_t N, uint32_t THREADS, uint32_t CAP, uint32_t LGB>
cudaError_t launch_unit_sort_t(const unsigned long long *tk, const uint32_t *tv, const unsigned long long *sub_off,
                               const unsigned long long *sub_final, const SubUnit *units, uint32_t n_units,
                               unsigned long long *out_k, uint32_t *out_v, uint64_t out_cap, cudaStream_t st)
{
    if (!n_units) return cudaSuccess;
    const size_t smem = (size_t)CAP * (8 * N + 2) + (size_t)(1u << LGB) * 4;
    auto kern = [] {
        if constexpr (N == 1) return k_unit_sort<THREADS, CAP, LGB>;
        else return k_unit_sort_wide<N, THREADS, CAP, LGB>;
    }();
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, THREADS, smem) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    note_kernel_launch();
    kern<<<std::min<uint32_t>(n_units, (uint32_t)(n_sms() * per_sm)), THREADS, smem, st>>>(
        tk, tv, sub_off, sub_final, units, n_units, out_k, out_v, out_cap);
    return cudaGetLastError();
}

template <uint32_t N>
cudaError_t launch_unit_sort_n(const unsigned long long *tk, const uint32_t *tv, const unsigned long long *sub_off,
                               const unsigned long long *sub_final, const SubUnit *units, const UnitLists &lists,
                               const uint32_t *n_units, unsigned long long *out_k, uint32_t *out_v, uint64_t out_cap,
                               cudaStream_t st)
{
    constexpr uint32_t C = unit_cap0(N);
    static_assert(UNIT_CLASSES == 4, "one launch per class");
    cudaError_t e = launch_unit_sort_t<N, 256, C, 9>(tk, tv, sub_off, sub_final, units + lists.base[0], n_units[0], out_k, out_v, out_cap,
                                                     st);
    if (e == cudaSuccess)
        e = launch_unit_sort_t<N, 256, 2 * C, 10>(tk, tv, sub_off, sub_final, units + lists.base[1], n_units[1], out_k, out_v,
                                                  out_cap, st);
    if (e == cudaSuccess)
        e = launch_unit_sort_t<N, 512, 4 * C, 11>(tk, tv, sub_off, sub_final, units + lists.base[2], n_units[2], out_k,
                                                  out_v, out_cap, st);
    if (e == cudaSuccess)
        e = launch_unit_sort_t<N, 512, 8 * C, 11>(tk, tv, sub_off, sub_final, units + lists.base[3], n_units[3], out_k,
                                                  out_v, out_cap, st);
    return e;
}

}  // namespace

cudaError_t launch_count_prefix(const PrefixCountArgs &a, uint32_t words, uint32_t shape, cudaStream_t st)
{
    if (!a.n_sub) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(a.next_sub, 0, 4, st);
    if (e != cudaSuccess) return e;
    const bool small = shape == 2 || shape == 4;
    if (words == 1) return small ? launch_count_prefix_t<1, 256, 4, 12>(a, st) : launch_count_prefix_t<1, 512, 2, 13>(a, st);
    if (words == 2) return small ? launch_count_prefix_t<2, 256, 4, 11>(a, st) : launch_count_prefix_t<2, 512, 2, 12>(a, st);
    return small ? launch_count_prefix_t<4, 256, 4, 10>(a, st) : launch_count_prefix_t<4, 512, 2, 11>(a, st);
}

cudaError_t launch_unit_sort(uint32_t words, const unsigned long long *tk, const uint32_t *tv,
                             const unsigned long long *sub_off, const unsigned long long *sub_final,
                             const SubUnit *units, const UnitLists &lists, const uint32_t *n_units,
                             unsigned long long *out_k, uint32_t *out_v, uint64_t out_cap, cudaStream_t st)
{
    if (words == 1)
        return launch_unit_sort_n<1>(tk, tv, sub_off, sub_final, units, lists, n_units, out_k, out_v, out_cap, st);
    if (words == 2)
        return launch_unit_sort_n<2>(tk, tv, sub_off, sub_final, units, lists, n_units, out_k, out_v, out_cap, st);
    return launch_unit_sort_n<4>(tk, tv, sub_off, sub_final, units, lists, n_units, out_k, out_v, out_cap, st);
}

}  // namespace kc
