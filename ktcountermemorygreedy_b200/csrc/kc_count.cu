// kc_count.cu -- counting of k-mers (k <= 32) by printed-order prefix, in
// shared memory, and the sort of the resulting records.
//
// The occurrences arrive partitioned twice, into 256 buckets by their first
// four bases and into sub-buckets by the next bases (launch_part by string,
// k_subpart_scatter), as string keys: the k bases first-base-high, left
// aligned.  So the sub-buckets are consecutive ranges of the printed order:
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
// min count 2) count 27.1 -> 18.5 ms and sort 7.1 -> 1.2 ms; 4M reads with
// every k-mer kept (480M k-mers, 145M records) insert + compaction 11.8 ms ->
// scatter + count 6.8 ms, sort 11.9 -> 1.7 ms.
#include <algorithm>

#include "kc_device.cuh"
#include "kc_kernels.cuh"

namespace kc {

namespace {

constexpr uint32_t FULLW = 0xffffffffu;
constexpr uint32_t CP_PER_THREAD = 4;       // keys per thread whose first probes are in flight together
constexpr uint32_t CP_HIST = 512;           // counts below this are histogrammed in shared memory
constexpr uint32_t CP_QUEUE = 64;           // keys a warp has waiting for their next probe
constexpr uint32_t CP_MAX_ROUNDS = 64;      // rounds a sub-bucket may be cut into

__device__ __forceinline__ uint32_t lanes_below()
{
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Placement hash of a key: two 32-bit multiplies over its halves (the top
// bits are the same for a whole sub-bucket, so the low half leads).  The top
// bits are its home slot, an odd number from the next ones its probe step.  It
// never affects a count.
__device__ __forceinline__ uint32_t mix_of(unsigned long long key)
{
    return ((uint32_t)key * 0x9E3779B1u + (uint32_t)(key >> 32)) * 0x85EBCA77u;
}

// Counts one sub-bucket per block at a time.  The keys are inserted into an
// open-addressing table in shared memory (a slot only changes from empty to a
// key, by CAS; no barrier between tiles): every key looks at its home slot,
// where most are found and counted; the others wait in the warp's queue until
// there are 32 of them, so that a probe step (claim, count, or on to the next
// slot and back into the queue) has all lanes busy.  (Each lane stepping its
// own keys to the end left 16 of 32 lanes active and 198 warp instructions per
// 32 keys; with the queue 23 and 172.  A ring that refilled each idle lane at
// every step took 248: more bookkeeping than probing.)  Bound by instruction
// issue (72%) and shared-memory wavefronts (63%): 2.4G k-mers of the 20M-read
// job 18.5 -> 15.6 ms, 480M k-mers with every record kept 3.8 -> 3.15, 25M
// mostly distinct ones 0.92 -> 0.49.  Then one sweep writes the kept
// records to the front of the sub-bucket's place in the record arrays,
// adds every count to the histogram and empties the table for the next
// sub-bucket.  A table that fills up (more distinct k-mers than it holds) is
// emptied and the sub-bucket counted in rounds over halves of its key range
// (quarters, ... at most CP_MAX_ROUNDS), each round reading the keys again
// from L2; a round's records lie after the earlier rounds' ones, and are a
// sort unit of their own.  The next sub-bucket's first keys are loaded before
// the sweep.
template <uint32_t THREADS, uint32_t BPSM, uint32_t TBITS>
__global__ void __launch_bounds__(THREADS, BPSM) k_count_prefix(PrefixCountArgs a)
{
    extern __shared__ __align__(16) uint8_t cp_smem[];
    unsigned long long *s_tk = reinterpret_cast<unsigned long long *>(cp_smem);   // 2^TBITS keys
    uint32_t *s_tc = reinterpret_cast<uint32_t *>(s_tk + (1u << TBITS));          // their counts
    uint32_t *s_hist = s_tc + (1u << TBITS);                                      // CP_HIST
    unsigned long long *q_key =                                                   // CP_QUEUE per warp
        reinterpret_cast<unsigned long long *>(s_hist + CP_HIST) + (threadIdx.x >> 5) * CP_QUEUE;
    uint16_t *q_slot = reinterpret_cast<uint16_t *>(s_hist + CP_HIST + 2 * CP_QUEUE * (THREADS / 32)) +
                       (threadIdx.x >> 5) * CP_QUEUE;
    __shared__ uint32_t s_out, s_full, s_next, s_next_n, s_next_plen;
    __shared__ unsigned long long s_next_off;
    constexpr uint32_t TILE_KEYS = THREADS * CP_PER_THREAD;
    const int tid = threadIdx.x, lane = tid & 31;
    const uint32_t lt = lanes_below();
    // sub-buckets that outgrew their regions are incomplete: nothing is counted
    if (a.counters[C_REGION_OVF]) return;
    for (uint32_t i = tid; i < (1u << TBITS); i += THREADS) {
        s_tk[i] = EMPTY_KEY;
        s_tc[i] = 0;
    }
    for (uint32_t i = tid; i < CP_HIST; i += THREADS) s_hist[i] = 0;
    uint32_t n_distinct = 0, n_once = 0, n_one = 0;   // per lane: below 2^32 whatever the pass
    unsigned long long n_kept = 0;
    uint32_t n_ovf_subs = 0, rounds0 = 1;
    bool unit_full = false;
    // thread 0 takes the next sub-bucket while this one is counted
    auto take_next = [&]() {
        const uint32_t s = atomicAdd(a.next_sub, 1u);
        s_next = s;
        if (s < a.n_sub) {
            s_next_n = a.sub_count[s];
            s_next_off = a.sub_off[s];
            s_next_plen = 8 + (31 - __clz(a.sc[a.sub_bucket[s]].n_sub));
        }
    };
    if (tid == 0) {
        s_out = 0;
        s_full = 0;
        take_next();
    }
    __syncthreads();
    unsigned long long kn[CP_PER_THREAD];
    uint32_t sub = s_next, n = 0, plen = 0;
    unsigned long long base = 0;
    if (sub < a.n_sub) {
        n = s_next_n;
        base = s_next_off;
        plen = s_next_plen;
#pragma unroll
        for (uint32_t r = 0; r < CP_PER_THREAD; ++r) {
            const uint32_t i = r * THREADS + tid;
            kn[r] = i < n ? __ldcs(&a.keys[base + i]) : EMPTY_KEY;
        }
    }
    while (sub < a.n_sub) {
        __syncthreads();   // s_next* read by all; the table is empty
        if (tid == 0) take_next();
        // slots for twice the keys where that is less than the whole table
        uint32_t lg = n > 1 ? 33 - __clz(n - 1) : 1;
        lg = lg < 9 ? 9 : (lg > TBITS ? TBITS : lg);
        const uint32_t smask = (1u << lg) - 1;
        uint32_t rounds = rounds0, rd = 0, off = 0, most = 0;
        bool failed = false;
        while (rd < rounds) {
            const uint32_t rmask = rounds - 1;
            const int rsh = 64 - (int)plen - (31 - __clz(rounds));   // rounds == 1: unused
            const bool reread = rd > 0 || failed;
            // a warp takes at most this many probe steps (a table less than
            // about five sixths full needs far fewer)
            const uint32_t hsh = 32 - lg;
            uint32_t qn = 0, steps = 0, most_steps = 3 * (n / THREADS + 1) + 64;
            // one more probe of the last `m` queued keys (m <= 32); those that
            // meet another key stay queued at their next slot
            auto probe_queue = [&](uint32_t m) {
                __syncwarp();
                qn -= m;
                ++steps;
                const bool in = lane < (int)m;
                unsigned long long key = 0;
                uint32_t slot = 0;
                bool wait = false;
                if (in) {
                    key = q_key[qn + lane];
                    slot = q_slot[qn + lane];
                    unsigned long long cur = *(volatile unsigned long long *)&s_tk[slot];
                    if (cur == EMPTY_KEY) {
                        cur = atomicCAS(&s_tk[slot], EMPTY_KEY, key);
                        if (cur == EMPTY_KEY) cur = key;   // claimed
                    }
                    wait = cur != key;
                    if (!wait) atomicAdd(&s_tc[slot], 1u);
                }
                const uint32_t w = __ballot_sync(FULLW, wait);
                if (wait) {
                    const uint32_t at = qn + (uint32_t)__popc(w & lt);
                    q_key[at] = key;
                    q_slot[at] = (uint16_t)((slot + (mix_of(key) >> 3 | 1u)) & smask);
                }
                qn += (uint32_t)__popc(w);
                __syncwarp();
            };
            for (uint32_t t0 = 0; t0 < n; t0 += TILE_KEYS) {
                unsigned long long k[CP_PER_THREAD];
                if (reread) {
#pragma unroll
                    for (uint32_t r = 0; r < CP_PER_THREAD; ++r) {
                        const uint32_t i = t0 + r * THREADS + tid;
                        k[r] = i < n ? __ldcg(&a.keys[base + i]) : EMPTY_KEY;
                    }
                } else {
#pragma unroll
                    for (uint32_t r = 0; r < CP_PER_THREAD; ++r) {
                        k[r] = kn[r];
                        const uint32_t i = t0 + TILE_KEYS + r * THREADS + tid;
                        kn[r] = i < n ? __ldcs(&a.keys[base + i]) : EMPTY_KEY;
                    }
                }
                if (rounds > 1) {
#pragma unroll
                    for (uint32_t r = 0; r < CP_PER_THREAD; ++r)
                        if (((uint32_t)(k[r] >> rsh) & rmask) != rd) k[r] = EMPTY_KEY;
                }
                // the home slots: most keys are there already and only counted
                uint32_t slot[CP_PER_THREAD];
                unsigned long long cur[CP_PER_THREAD];
#pragma unroll
                for (uint32_t r = 0; r < CP_PER_THREAD; ++r) {
                    slot[r] = mix_of(k[r]) >> hsh;
                    cur[r] = *(volatile unsigned long long *)&s_tk[slot[r]];
                }
#pragma unroll
                for (uint32_t r = 0; r < CP_PER_THREAD; ++r) {
                    const bool in = k[r] != EMPTY_KEY, hit = in && cur[r] == k[r];
                    if (hit) atomicAdd(&s_tc[slot[r]], 1u);
                    const uint32_t w = __ballot_sync(FULLW, in && !hit);
                    if (in && !hit) {
                        const uint32_t at = qn + (uint32_t)__popc(w & lt);
                        q_key[at] = k[r];
                        q_slot[at] = (uint16_t)slot[r];
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
                    s_tk[i] = EMPTY_KEY;
                    s_tc[i] = 0;
                }
                if (tid == 0) s_full = 0;
                __syncthreads();
                failed = true;
                rounds *= 2;
                rd *= 2;
                if (rounds > CP_MAX_ROUNDS || (int)plen + (31 - __clz(rounds)) > 64) break;
                continue;
            }
            if (rd + 1 == rounds) {
                // the next sub-bucket's first keys arrive during the sweep
                const uint32_t nn = s_next < a.n_sub ? s_next_n : 0u;
#pragma unroll
                for (uint32_t r = 0; r < CP_PER_THREAD; ++r) {
                    const uint32_t i = r * THREADS + tid;
                    kn[r] = i < nn ? __ldcs(&a.keys[s_next_off + i]) : EMPTY_KEY;
                }
            }
            // the sweep: records out, histogram, table emptied
            const unsigned long long out = base + off;
            for (uint32_t i0 = 0; i0 <= smask; i0 += 2 * THREADS) {
                const uint32_t i = i0 + 2 * tid;   // two slots a thread
                ulonglong2 kk = make_ulonglong2(EMPTY_KEY, EMPTY_KEY);
                uint32_t c[2] = {0, 0};
                bool keep[2] = {false, false};
                if (i <= smask) kk = *reinterpret_cast<const ulonglong2 *>(&s_tk[i]);
                const unsigned long long key[2] = {kk.x, kk.y};
                if (kk.x != EMPTY_KEY || kk.y != EMPTY_KEY) {
                    const uint2 raw2 = *reinterpret_cast<const uint2 *>(&s_tc[i]);
                    *reinterpret_cast<ulonglong2 *>(&s_tk[i]) = make_ulonglong2(EMPTY_KEY, EMPTY_KEY);
                    *reinterpret_cast<uint2 *>(&s_tc[i]) = make_uint2(0u, 0u);
                    const uint32_t raw[2] = {raw2.x, raw2.y};
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        if (key[j] == EMPTY_KEY) continue;
                        ++n_distinct;
                        n_once += raw[j] == 1;
                        c[j] = raw[j] < a.count_max ? raw[j] : a.count_max;
                        if (c[j] == 1) ++n_one;   // most k-mers of many inputs: one shared bin would serialize
                        else if (c[j] < CP_HIST) atomicAdd(&s_hist[c[j]], 1u);
                        else if (c[j] < HIST_BINS) atomicAdd(&a.hist[c[j]], 1ull);
                        else {
                            const unsigned long long q = atomicAdd(&a.counters[C_OVF_LEN], 1ull);
                            if (q < a.ovf_cap) a.ovf[q] = c[j];
                            else atomicOr(&a.counters[C_FLAGS], ERR_HIST_OVERFLOW_FULL);
                        }
                        keep[j] = c[j] >= a.min_count && c[j] <= a.max_count;
                    }
                }
                const uint32_t b0 = __ballot_sync(FULLW, keep[0]), b1 = __ballot_sync(FULLW, keep[1]);
                if (b0 | b1) {
                    uint32_t w = 0;
                    if (lane == 0) w = atomicAdd(&s_out, (uint32_t)(__popc(b0) + __popc(b1)));
                    w = __shfl_sync(FULLW, w, 0);
                    if (keep[0]) {
                        const unsigned long long q = out + w + (uint32_t)__popc(b0 & lt);
                        a.rec_keys[q] = key[0];
                        a.rec_counts[q] = c[0];
                    }
                    if (keep[1]) {
                        const unsigned long long q = out + w + (uint32_t)(__popc(b0) + __popc(b1 & lt));
                        a.rec_keys[q] = key[1];
                        a.rec_counts[q] = c[1];
                    }
                }
            }
            __syncthreads();
            const uint32_t len = s_out;
            __syncthreads();
            if (tid == 0) {
                s_out = 0;
                if (len) {
                    const uint32_t cls = len <= UNIT_CAP0 ? 0 : (len <= 2 * UNIT_CAP0 ? 1 : (len <= 4 * UNIT_CAP0 ? 2 : 3));
                    const unsigned long long u = atomicAdd(&a.counters[C_UNITS + cls], 1ull);
                    if (u < a.unit_cap) a.units[cls * (uint64_t)a.unit_cap + u] = SubUnit{sub, off, len, 0u};
                    else unit_full = true;
                    n_kept += len;
                }
            }
            off += len;
            most = len > most ? len : most;
            ++rd;
        }
        const bool gave_up = rd < rounds;   // uniform
        if (tid == 0) {
            a.sub_len[sub] = off;
            if (gave_up) {
                ++n_ovf_subs;
                atomicOr(&a.bucket_ovf[a.sub_bucket[sub]], 1u);
            }
        }
        // sub-buckets are alike: the next one starts with as many rounds,
        // or with half as many when no round came near the table's size
        rounds0 = gave_up ? 1u : (rounds > 1 && most < (1u << TBITS) / 4 ? rounds / 2 : rounds);
        if (gave_up) {
            const uint32_t nn = s_next < a.n_sub ? s_next_n : 0u;
#pragma unroll
            for (uint32_t r = 0; r < CP_PER_THREAD; ++r) {
                const uint32_t i = r * THREADS + tid;
                kn[r] = i < nn ? __ldcs(&a.keys[s_next_off + i]) : EMPTY_KEY;
            }
        }
        sub = s_next;
        n = s_next_n;
        base = s_next_off;
        plen = s_next_plen;
    }
    __syncthreads();
    for (uint32_t i = tid; i < CP_HIST; i += THREADS)
        if (s_hist[i]) atomicAdd(&a.hist[i], (unsigned long long)s_hist[i]);
    if (tid == 0 && unit_full) n_ovf_subs += 1;   // more sort units than the lists hold: counted as an overflow
    unsigned long long s[4] = {n_distinct, n_once, n_one, n_kept};
#pragma unroll
    for (int j = 0; j < 4; ++j)
        for (int o = 16; o > 0; o >>= 1) s[j] += __shfl_down_sync(FULLW, s[j], o);
    if (lane == 0) {
        if (s[0]) atomicAdd(&a.counters[C_DISTINCT], s[0]);
        if (s[1]) atomicAdd(&a.counters[C_LOW_ONLY], s[1]);
        if (s[2]) atomicAdd(&a.hist[1], s[2]);
        if (s[3]) atomicAdd(&a.counters[C_REC_LEN], s[3]);
    }
    if (tid == 0 && n_ovf_subs) atomicAdd(&a.counters[C_SUB_OVF], (unsigned long long)n_ovf_subs);
}

// Sorts the records of one unit (a sub-bucket, or one round of it: at most
// CAP records of one range of the printed order) per block at a time and
// writes them, as k-mer words, to their final place.  The keys come into
// shared memory once; their indexes are placed by the 2^LGB values of the bits
// below the unit's common prefix (the xor of all its keys says where that
// ends), then each record finds its rank inside its run of a few records by
// comparing itself with the run's other keys: no lane waits for another,
// unlike an insertion sort per run.  The counts are read where they are
// written (a unit's counts stay in L1).
template <uint32_t THREADS, uint32_t CAP, uint32_t LGB>
__global__ void __launch_bounds__(THREADS) k_unit_sort(const unsigned long long *tk, const uint32_t *tv,
                                                       const unsigned long long *sub_off,
                                                       const unsigned long long *sub_final, const SubUnit *units,
                                                       uint32_t n_units, unsigned long long *out_k, uint32_t *out_v,
                                                       uint64_t out_cap, uint32_t kshift)
{
    constexpr uint32_t NB = 1u << LGB, PER = NB / THREADS, WARPS = THREADS / 32;
    static_assert(NB % THREADS == 0 && CAP <= 65536, "layout");
    extern __shared__ __align__(16) uint8_t us_smem[];
    unsigned long long *s_keys = reinterpret_cast<unsigned long long *>(us_smem);   // CAP
    uint32_t *s_start = reinterpret_cast<uint32_t *>(s_keys + CAP);                 // NB + 1 (+ 3: alignment)
    uint16_t *s_idx = reinterpret_cast<uint16_t *>(s_start + NB + 4);               // CAP
    __shared__ uint32_t s_warp[WARPS], s_xlo, s_xhi;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (uint32_t ui = blockIdx.x; ui < n_units; ui += gridDim.x) {
        const SubUnit u = units[ui];
        const uint32_t m = u.len < CAP ? u.len : CAP;
        const unsigned long long src = sub_off[u.sub] + u.off, dst = sub_final[u.sub] + u.off;
        if (tid == 0) {
            s_xlo = s_xhi = 0;
            s_start[NB] = m;
        }
#pragma unroll
        for (uint32_t j = 0; j < PER; ++j) s_start[j * THREADS + tid] = 0;
        __syncthreads();
        // common prefix: the bits in which no key differs from the first
        const unsigned long long k0 = __ldg(&tk[src]);
        unsigned long long x = 0;
#pragma unroll 4
        for (uint32_t i = tid; i < m; i += THREADS) {
            const unsigned long long key = __ldcs(&tk[src + i]);
            s_keys[i] = key;
            x |= key ^ k0;
        }
        const uint32_t xh = __reduce_or_sync(FULLW, (uint32_t)(x >> 32)), xl = __reduce_or_sync(FULLW, (uint32_t)x);
        if (lane == 0) {
            if (xh) atomicOr(&s_xhi, xh);
            if (xl) atomicOr(&s_xlo, xl);
        }
        __syncthreads();
        const int pre = __clzll(((unsigned long long)s_xhi << 32) | s_xlo);   // 64: one record
        const int dsh = 64 - pre - (int)LGB > 0 ? 64 - pre - (int)LGB : 0;
        for (uint32_t i = tid; i < m; i += THREADS) atomicAdd(&s_start[(uint32_t)(s_keys[i] >> dsh) & (NB - 1)], 1u);
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
        for (uint32_t i = tid; i < m; i += THREADS)
            s_idx[atomicAdd(&s_start[(uint32_t)(s_keys[i] >> dsh) & (NB - 1)], 1u)] = (uint16_t)i;
        __syncthreads();
        for (uint32_t p = tid; p < m; p += THREADS) {
            const uint32_t i = s_idx[p];
            const unsigned long long key = s_keys[i];
            const uint32_t d = (uint32_t)(key >> dsh) & (NB - 1);
            const uint32_t lo = d ? s_start[d - 1] : 0u, hi = s_start[d];
            uint32_t rank = lo;
            for (uint32_t j = lo; j < hi; ++j) rank += s_keys[s_idx[j]] < key ? 1u : 0u;
            if (dst + rank < out_cap) {
                out_k[dst + rank] = pair_reverse(key) << kshift;
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

template <uint32_t THREADS, uint32_t BPSM, uint32_t TBITS>
cudaError_t launch_count_prefix_t(const PrefixCountArgs &a, cudaStream_t st)
{
    const size_t smem = ((size_t)1 << TBITS) * 12 + CP_HIST * 4 + (THREADS / 32) * CP_QUEUE * 10;
    auto kern = k_count_prefix<THREADS, BPSM, TBITS>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    note_kernel_launch();
    kern<<<std::min<uint32_t>(a.n_sub, (uint32_t)n_sms() * BPSM), THREADS, smem, st>>>(a);
    return cudaGetLastError();
}

template <uint32_t THREADS, uint32_t CAP, uint32_t LGB>
cudaError_t launch_unit_sort_t(const unsigned long long *tk, const uint32_t *tv, const unsigned long long *sub_off,
                               const unsigned long long *sub_final, const SubUnit *units, uint32_t n_units,
                               unsigned long long *out_k, uint32_t *out_v, uint64_t out_cap, uint32_t k, cudaStream_t st)
{
    if (!n_units) return cudaSuccess;
    const size_t smem = (size_t)CAP * 10 + ((size_t)(1u << LGB) + 4) * 4;
    auto kern = k_unit_sort<THREADS, CAP, LGB>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, THREADS, smem) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    note_kernel_launch();
    kern<<<std::min<uint32_t>(n_units, (uint32_t)(n_sms() * per_sm)), THREADS, smem, st>>>(
        tk, tv, sub_off, sub_final, units, n_units, out_k, out_v, out_cap, 64 - 2 * k);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_count_prefix(const PrefixCountArgs &a, uint32_t shape, cudaStream_t st)
{
    if (!a.n_sub) return cudaSuccess;
    cudaError_t e = cudaMemsetAsync(a.next_sub, 0, 4, st);
    if (e != cudaSuccess) return e;
    return (shape == 2 || shape == 4) ? launch_count_prefix_t<256, 4, 12>(a, st) : launch_count_prefix_t<512, 2, 13>(a, st);
}

cudaError_t launch_unit_sort(const unsigned long long *tk, const uint32_t *tv, const unsigned long long *sub_off,
                             const unsigned long long *sub_final, const SubUnit *units, uint32_t unit_cap,
                             const uint32_t *n_units, unsigned long long *out_k, uint32_t *out_v, uint64_t out_cap,
                             uint32_t k, cudaStream_t st)
{
    static_assert(UNIT_CAP0 == 1024 && UNIT_CLASSES == 4, "one launch per class");
    cudaError_t e = launch_unit_sort_t<256, 1024, 9>(tk, tv, sub_off, sub_final, units, n_units[0], out_k, out_v, out_cap,
                                                     k, st);
    if (e == cudaSuccess)
        e = launch_unit_sort_t<256, 2048, 10>(tk, tv, sub_off, sub_final, units + unit_cap, n_units[1], out_k, out_v,
                                              out_cap, k, st);
    if (e == cudaSuccess)
        e = launch_unit_sort_t<512, 4096, 11>(tk, tv, sub_off, sub_final, units + 2ull * unit_cap, n_units[2], out_k,
                                              out_v, out_cap, k, st);
    if (e == cudaSuccess)
        e = launch_unit_sort_t<512, 8192, 11>(tk, tv, sub_off, sub_final, units + 3ull * unit_cap, n_units[3], out_k,
                                              out_v, out_cap, k, st);
    return e;
}

}  // namespace kc
