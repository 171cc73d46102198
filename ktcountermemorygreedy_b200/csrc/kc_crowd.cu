// kc_crowd.cu -- the crowded sub-buckets of a counting pass by printed-order
// prefix: those whose distinct k-mers fit a shared-memory table in no number of
// rounds (rounds tell k-mers apart by their first bases only, and poly-A,
// microsatellites or the errors of a deeply sequenced amplicon share many of
// those), or whose occurrences would keep one block busy for milliseconds.
//
// Their keys lie together in sub-bucket order.  What their finished rounds have
// not counted is gathered, sorted by whole key and counted as runs of equal keys:
// no table, so it does not matter how the keys are spread, and every thread block
// takes part whatever the sub-bucket's size.  The records go behind those of the
// sub-bucket's finished rounds, in order, and from there to their final place.
//
// When such sub-buckets sent the whole job (or batch) to global-memory tables: 960M
// 31-mers of a 40 Mbp genome with 1% of poly-A and microsatellites 477 ms a call,
// now 19.5 (17 crowded sub-buckets, 7.7M keys, 1.3 ms of it here; 17.1 without the
// repeats), 176M 63-mers 73 -> 10.8, 48 samples with one of repeats 84 -> 18.4.
#include <algorithm>

#include "kc_device.cuh"
#include "kc_kernels.cuh"

namespace kc {

namespace {

constexpr uint32_t FULLW = 0xffffffffu;
constexpr uint32_t CROWD_THREADS = 256, CROWD_PER_THREAD = 4;
constexpr uint32_t CROWD_HIST = 512;   // counts below this are histogrammed in shared memory

// The last of n ranges whose start is at or before i.
template <class R>
__device__ __forceinline__ uint32_t range_of(const R *r, uint32_t n, unsigned long long i)
{
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (r[mid].start <= i) lo = mid;
        else hi = mid;
    }
    return lo;
}

// A key as it is sorted: one word, right aligned; more words, as k-mer words
// (word w holds the 32 bases ending 32w before the last, newest at the top).
template <uint32_t N>
__device__ __forceinline__ void to_sorted_form(const unsigned long long *s, uint32_t k, unsigned long long *out)
{
    if constexpr (N == 1) {
        out[0] = s[0] >> (64 - 2 * k);
    } else {
        for (uint32_t w = 0; w < N; ++w) {
            const int b = (int)k - 32 * (int)(w + 1);   // first base of the word
            unsigned long long v = 0;
            if (b >= 0) {
                const uint32_t o = 2 * (b & 31), q = (uint32_t)b >> 5;
                v = s[q] << o;
                if (o) v |= s[q + 1] >> (64 - o);
            } else if (b > -32) {
                v = s[0] >> (-2 * b);
            }
            out[w] = pair_reverse(v);
        }
    }
}

// The keys that the finished rounds left, in any order, each with its range's
// number.
template <uint32_t N>
__global__ void __launch_bounds__(CROWD_THREADS) k_crowd_gather(const unsigned long long *keys, const CrowdRange *rg,
                                                                uint32_t n_rg, unsigned long long total, uint32_t k,
                                                                unsigned long long *out, uint32_t *out_range,
                                                                unsigned long long *cursor)
{
    const uint32_t lane = threadIdx.x & 31;
    const unsigned long long step = (unsigned long long)gridDim.x * CROWD_THREADS * CROWD_PER_THREAD;
    for (unsigned long long i0 = (unsigned long long)blockIdx.x * CROWD_THREADS * CROWD_PER_THREAD; i0 < total; i0 += step) {
        unsigned long long key[CROWD_PER_THREAD][N];
        uint32_t at[CROWD_PER_THREAD];
        uint32_t j[CROWD_PER_THREAD], n = 0;
        bool take[CROWD_PER_THREAD];
#pragma unroll
        for (uint32_t r = 0; r < CROWD_PER_THREAD; ++r) {
            const unsigned long long i = i0 + r * CROWD_THREADS + threadIdx.x;
            take[r] = false;
            if (i < total) {
                j[r] = range_of(rg, n_rg, i);
                const CrowdRange c = rg[j[r]];
                const unsigned long long *p = keys + (c.src + (i - c.start)) * N;
#pragma unroll
                for (uint32_t w = 0; w < N; ++w) key[r][w] = p[w];
                take[r] = c.rd == 0 || ((uint32_t)(key[r][0] >> c.shift) & c.mask) >= c.rd;
            }
            const uint32_t b = __ballot_sync(FULLW, take[r]);
            at[r] = n + (uint32_t)__popc(b & ((1u << lane) - 1u));
            n += (uint32_t)__popc(b);
        }
        unsigned long long base = 0;
        if (lane == 0 && n) base = atomicAdd(cursor, (unsigned long long)n);
        base = __shfl_sync(FULLW, base, 0);
#pragma unroll
        for (uint32_t r = 0; r < CROWD_PER_THREAD; ++r)
            if (take[r]) {
                to_sorted_form<N>(key[r], k, out + (base + at[r]) * N);
                out_range[base + at[r]] = j[r];
            }
    }
}

template <uint32_t N>
__global__ void __launch_bounds__(CROWD_THREADS) k_crowd_heads(const unsigned long long *keys, uint64_t m, uint32_t *head)
{
    for (uint64_t i = blockIdx.x * (uint64_t)CROWD_THREADS + threadIdx.x; i < m; i += (uint64_t)gridDim.x * CROWD_THREADS) {
        bool h = i == 0;
        if (!h) {
#pragma unroll
            for (uint32_t w = 0; w < N; ++w) h = h || keys[i * N + w] != keys[(i - 1) * N + w];
        }
        head[i] = h ? 1u : 0u;
    }
}

// start[r] = first key of run r; start[number of runs] = m.
__global__ void __launch_bounds__(CROWD_THREADS) k_crowd_starts(const uint32_t *head, const unsigned long long *run,
                                                                uint64_t m, uint32_t *start)
{
    for (uint64_t i = blockIdx.x * (uint64_t)CROWD_THREADS + threadIdx.x; i < m; i += (uint64_t)gridDim.x * CROWD_THREADS) {
        if (head[i]) start[run[i]] = (uint32_t)i;
        if (i == m - 1) start[run[i] + head[i]] = (uint32_t)m;
    }
}

// Histogram and totals of every run; keep[i] = 1 at the first key of each run
// that is a record.
__global__ void __launch_bounds__(CROWD_THREADS) k_crowd_runs(const uint32_t *head, const unsigned long long *run,
                                                              const uint32_t *start, uint64_t m, SubCfg c, uint32_t *keep,
                                                              PrefixCountArgs a)
{
    __shared__ uint32_t s_hist[CROWD_HIST];
    for (uint32_t i = threadIdx.x; i < CROWD_HIST; i += CROWD_THREADS) s_hist[i] = 0;
    __syncthreads();
    unsigned long long *hist = a.hist + (unsigned long long)c.group * a.hist_bins;
    unsigned long long t[4] = {0, 0, 0, 0};   // distinct, seen once, records, counts of 1
    for (uint64_t i = blockIdx.x * (uint64_t)CROWD_THREADS + threadIdx.x; i < m; i += (uint64_t)gridDim.x * CROWD_THREADS) {
        bool kept = false;
        if (head[i]) {
            const uint32_t raw = start[run[i] + 1] - (uint32_t)i, n = raw < c.count_max ? raw : c.count_max;
            ++t[0];
            t[1] += raw == 1;
            if (n == 1) ++t[3];
            else if (n < CROWD_HIST) atomicAdd(&s_hist[n], 1u);
            else if (n < a.hist_bins) atomicAdd(&hist[n], 1ull);
            else {
                const unsigned long long q = atomicAdd(&a.counters[C_OVF_LEN], 1ull);
                if (q >= a.ovf_cap) atomicOr(&a.counters[C_FLAGS], ERR_HIST_OVERFLOW_FULL);
                else if (a.ovf64) a.ovf64[q] = ((unsigned long long)c.group << 32) | n;
                else a.ovf[q] = n;
            }
            kept = n >= c.min_count && n <= c.max_count;
            t[2] += kept;
        }
        keep[i] = kept ? 1u : 0u;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        for (int o = 16; o > 0; o >>= 1) t[j] += __shfl_down_sync(FULLW, t[j], o);
        if ((threadIdx.x & 31) == 0 && t[j]) atomicAdd(j < 3 ? &a.totals[3ull * c.group + j] : &hist[1], t[j]);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < CROWD_HIST; i += CROWD_THREADS)
        if (s_hist[i]) atomicAdd(&hist[i], (unsigned long long)s_hist[i]);
}

// first[j] = records before range j's; first[n_rg] = all records.
__global__ void __launch_bounds__(CROWD_THREADS) k_crowd_first(const uint32_t *range, const uint32_t *keep,
                                                               const unsigned long long *rec, uint64_t m, uint32_t n_rg,
                                                               unsigned long long *first)
{
    for (uint64_t i = blockIdx.x * (uint64_t)CROWD_THREADS + threadIdx.x; i < m; i += (uint64_t)gridDim.x * CROWD_THREADS) {
        if (i == 0 || range[i] != range[i - 1]) first[range[i]] = rec[i];
        if (i == m - 1) first[n_rg] = rec[i] + keep[i];
    }
}

// Records, as k-mer words, to the end of their sub-bucket's place.
template <uint32_t N>
__global__ void __launch_bounds__(CROWD_THREADS) k_crowd_place(const unsigned long long *keys, const uint32_t *range,
                                                               const unsigned long long *run, const uint32_t *start,
                                                               const uint32_t *keep, const unsigned long long *rec,
                                                               const unsigned long long *first, uint64_t m,
                                                               const CrowdRange *rg, uint32_t count_max,
                                                               unsigned long long *rec_keys, uint32_t *rec_counts)
{
    for (uint64_t i = blockIdx.x * (uint64_t)CROWD_THREADS + threadIdx.x; i < m; i += (uint64_t)gridDim.x * CROWD_THREADS) {
        if (!keep[i]) continue;
        const uint32_t raw = start[run[i] + 1] - (uint32_t)i, j = range[i];
        const unsigned long long at = rg[j].src + rg[j].off + (rec[i] - first[j]);
#pragma unroll
        for (uint32_t w = 0; w < N; ++w) {
            const unsigned long long x = keys[i * N + w];
            rec_keys[at * N + w] = N == 1 ? pair_reverse(x) : x;
        }
        rec_counts[at] = raw < count_max ? raw : count_max;
    }
}

__global__ void k_crowd_lens(const CrowdRecords *r, uint32_t n, uint32_t *sub_len)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) sub_len[r[i].sub] += r[i].len;
}

template <uint32_t N>
__global__ void __launch_bounds__(CROWD_THREADS) k_crowd_copy(const CrowdRecords *r, uint32_t n_r, unsigned long long total,
                                                              const unsigned long long *rec_keys, const uint32_t *rec_counts,
                                                              const unsigned long long *sub_final, unsigned long long *out_k,
                                                              uint32_t *out_v, uint64_t out_cap)
{
    for (unsigned long long i = blockIdx.x * (unsigned long long)CROWD_THREADS + threadIdx.x; i < total;
         i += (unsigned long long)gridDim.x * CROWD_THREADS) {
        const CrowdRecords c = r[range_of(r, n_r, i)];
        const unsigned long long s = c.src + (i - c.start), d = sub_final[c.sub] + c.off + (i - c.start);
        if (d >= out_cap) continue;
#pragma unroll
        for (uint32_t w = 0; w < N; ++w) out_k[d * N + w] = rec_keys[s * N + w];
        out_v[d] = rec_counts[s];
    }
}

inline unsigned crowd_grid(uint64_t n) { return (unsigned)std::min<uint64_t>((n + CROWD_THREADS - 1) / CROWD_THREADS, 148 * 8); }
inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

template <uint32_t N>
cudaError_t gather(const unsigned long long *keys, const CrowdRange *rg, uint32_t n_rg, uint64_t total, uint32_t k,
                   unsigned long long *out, uint32_t *out_range, unsigned long long *cursor, cudaStream_t st)
{
    note_kernel_launch();
    k_crowd_gather<N><<<crowd_grid((total + CROWD_PER_THREAD - 1) / CROWD_PER_THREAD), CROWD_THREADS, 0, st>>>(
        keys, rg, n_rg, total, k, out, out_range, cursor);
    return cudaGetLastError();
}

template <uint32_t N>
cudaError_t runs(const unsigned long long *keys, const uint32_t *range, uint64_t m, const CrowdRange *rg, uint32_t n_rg,
                 const SubCfg &c, const PrefixCountArgs &a, void *tmp, unsigned long long *first, cudaStream_t st)
{
    uint8_t *p = static_cast<uint8_t *>(tmp);
    uint32_t *head = reinterpret_cast<uint32_t *>(p);
    p += align256(m * 4);
    uint32_t *keep = reinterpret_cast<uint32_t *>(p);
    p += align256(m * 4);
    uint32_t *start = reinterpret_cast<uint32_t *>(p);
    p += align256((m + 1) * 4);
    unsigned long long *run = reinterpret_cast<unsigned long long *>(p);
    p += align256(m * 8);
    unsigned long long *rec = reinterpret_cast<unsigned long long *>(p);
    p += align256(m * 8);
    unsigned long long *stmp = reinterpret_cast<unsigned long long *>(p);
    const unsigned g = crowd_grid(m);
    note_kernel_launch();
    k_crowd_heads<N><<<g, CROWD_THREADS, 0, st>>>(keys, m, head);
    cudaError_t e = launch_scan_u32(head, run, m, stmp, st);
    if (e != cudaSuccess) return e;
    note_kernel_launch();
    k_crowd_starts<<<g, CROWD_THREADS, 0, st>>>(head, run, m, start);
    note_kernel_launch();
    k_crowd_runs<<<g, CROWD_THREADS, 0, st>>>(head, run, start, m, c, keep, a);
    e = launch_scan_u32(keep, rec, m, stmp, st);
    if (e != cudaSuccess) return e;
    note_kernel_launch();
    k_crowd_first<<<g, CROWD_THREADS, 0, st>>>(range, keep, rec, m, n_rg, first);
    note_kernel_launch();
    k_crowd_place<N><<<g, CROWD_THREADS, 0, st>>>(keys, range, run, start, keep, rec, first, m, rg, c.count_max, a.rec_keys,
                                                  a.rec_counts);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_crowd_gather(uint32_t words, const unsigned long long *keys, const CrowdRange *rg, uint32_t n_rg,
                                uint64_t total, uint32_t k, unsigned long long *out, uint32_t *out_range,
                                unsigned long long *cursor, cudaStream_t st)
{
    if (!total || !n_rg) return cudaSuccess;
    if (words == 1) return gather<1>(keys, rg, n_rg, total, k, out, out_range, cursor, st);
    if (words == 2) return gather<2>(keys, rg, n_rg, total, k, out, out_range, cursor, st);
    return gather<4>(keys, rg, n_rg, total, k, out, out_range, cursor, st);
}

size_t crowd_runs_tmp_bytes(uint64_t m)
{
    return 2 * align256(m * 4) + align256((m + 1) * 4) + 2 * align256(m * 8) + align256(scan_tmp_words(m) * 8);
}

cudaError_t launch_crowd_runs(uint32_t words, const unsigned long long *keys, const uint32_t *range, uint64_t m,
                              const CrowdRange *rg, uint32_t n_rg, const SubCfg &c, const PrefixCountArgs &a, void *tmp,
                              unsigned long long *first, cudaStream_t st)
{
    if (!m) return cudaSuccess;
    if (m >= 0xFFFFFFFFull) return cudaErrorInvalidValue;   // run starts take 32 bits
    if (words == 1) return runs<1>(keys, range, m, rg, n_rg, c, a, tmp, first, st);
    if (words == 2) return runs<2>(keys, range, m, rg, n_rg, c, a, tmp, first, st);
    return runs<4>(keys, range, m, rg, n_rg, c, a, tmp, first, st);
}

cudaError_t launch_crowd_lens(const CrowdRecords *r, uint32_t n, uint32_t *sub_len, cudaStream_t st)
{
    if (!n) return cudaSuccess;
    note_kernel_launch();
    k_crowd_lens<<<crowd_grid(n), CROWD_THREADS, 0, st>>>(r, n, sub_len);
    return cudaGetLastError();
}

cudaError_t launch_crowd_copy(uint32_t words, const CrowdRecords *r, uint32_t n_r, uint64_t total,
                              const unsigned long long *rec_keys, const uint32_t *rec_counts,
                              const unsigned long long *sub_final, unsigned long long *out_k, uint32_t *out_v,
                              uint64_t out_cap, cudaStream_t st)
{
    if (!total || !n_r) return cudaSuccess;
    note_kernel_launch();
    const unsigned g = crowd_grid(total);
    if (words == 1)
        k_crowd_copy<1><<<g, CROWD_THREADS, 0, st>>>(r, n_r, total, rec_keys, rec_counts, sub_final, out_k, out_v, out_cap);
    else if (words == 2)
        k_crowd_copy<2><<<g, CROWD_THREADS, 0, st>>>(r, n_r, total, rec_keys, rec_counts, sub_final, out_k, out_v, out_cap);
    else
        k_crowd_copy<4><<<g, CROWD_THREADS, 0, st>>>(r, n_r, total, rec_keys, rec_counts, sub_final, out_k, out_v, out_cap);
    return cudaGetLastError();
}

}  // namespace kc
